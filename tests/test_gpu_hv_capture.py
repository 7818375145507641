"""FP64 products captured into CUDA graphs from the context's stream.

Each captured product depends on its own vectors and the uploaded superblock
alone, so graphs of one superblock may be replayed on several streams at once.
The replays have to give, bit for bit, what one of them alone gives; that one
is held to a chain of FP64 additions: 2 (Dl + Dr + 2) 2^-53 sum |a||b|.
"""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("split", ["0", "1"])
@pytest.mark.parametrize("dims", [[(60, 60)] * 40, [(130, 70), (33, 200)]], ids=lambda d: f"{len(d)}x{d[0]}")
def test_replays_at_the_same_time(monkeypatch, dims, split):
    import torch

    import nssdmrg_gb300 as nss
    nss.lib()
    monkeypatch.setenv("NSS_SPLIT64", split)
    rng = np.random.default_rng(len(dims))
    hl, hr = [[rng.standard_normal((d[i], d[i])) for d in dims] for i in (0, 1)]
    off = np.concatenate([[0], np.cumsum([a * b for a, b in dims])[:-1]]).astype(np.int64)
    s = nss.Superblock()
    s.upload([a for a, _ in dims], [b for _, b in dims], off, [sp.csr_matrix(h) for h in hl],
             [sp.csr_matrix(h) for h in hr], [], 0, sum(a for a, _ in dims), sum(b for _, b in dims))
    vs = [torch.from_numpy(rng.standard_normal(s.n)).cuda() for _ in range(3)]
    outs = [torch.zeros_like(v) for v in vs]
    own = torch.cuda.ExternalStream(s.stream)
    graphs = []
    torch.cuda.synchronize()
    for v, o in zip(vs, outs):
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=own, capture_error_mode="thread_local"):
            s.hv_device(v.data_ptr(), o.data_ptr())
        graphs.append(g)
    streams = [torch.cuda.Stream() for _ in graphs]
    alone = []
    for g, o in zip(graphs, outs):
        g.replay()
        torch.cuda.synchronize()
        alone.append(o.clone())
    for v, w in zip(vs, alone):
        v, w = v.cpu().numpy(), w.cpu().numpy()
        for k, (a, b) in enumerate(dims):
            W, got = (x[off[k]:off[k] + a * b].reshape(a, b) for x in (v, w))
            mag = abs(hl[k]) @ abs(W) + abs(W) @ abs(hr[k].T)
            assert (abs(got - (hl[k] @ W + W @ hr[k].T)) <= 2 * (a + b + 2) * 2.0 ** -53 * mag).all()
    for _ in range(20):
        for o in outs:
            o.zero_()
        torch.cuda.synchronize()
        for g, st in zip(graphs, streams):
            with torch.cuda.stream(st):
                g.replay()
        torch.cuda.synchronize()
        for o, w in zip(outs, alone):
            assert torch.equal(o, w)
    # a product of the context itself beside them
    s.spmatvec(vs[0].cpu().numpy())
    del graphs
    s.close()
