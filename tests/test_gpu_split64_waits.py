"""A tensor-core FP64 product whose waits run out.

NSS_WAIT_LIMIT=0 (a test knob) makes every bounded wait of k_sector_split give
up after its first poll: the kernel returns without its sums.  nss_hv and
nss_hv_device must give the right product all the same (k_hv_fp64 computes it),
and the context works afterwards.
"""
import numpy as np
import pytest

from conftest import load_npz
from oracle import dmrg_oracle as O
from tests.golden.blockio import unpack_block

pytestmark = pytest.mark.gpu


def _upload(monkeypatch, split):
    import nssdmrg_gb300 as nss
    nss.lib()
    monkeypatch.setenv("NSS_SPLIT64", split)
    z = load_npz("c2_small.npz")
    l, r = unpack_block("eleft", z), unpack_block("eright", z)
    sb = O.sb_get_states(l, r, z["target"])
    ds = O.setup_direct(l, r, sb, z["hij"])
    terms = [(t.it - 1, t.isb, t.jsb, t.hconj, t.A, t.B, t.row_offset, t.col_offset) for t in ds.terms]
    s = nss.Superblock()
    s.upload(sb.Dls, sb.Drs, sb.Offset, ds.Hleft, ds.Hright, terms, ds.tNso, l.dim, r.dim, sb.AI, sb.BI)
    return nss, s, z["oracle_gs_energy"][0]


def test_product_is_right_when_its_waits_run_out(monkeypatch):
    import torch
    nss, s, _ = _upload(monkeypatch, "1")
    _, g, _ = _upload(monkeypatch, "0")
    rng = np.random.default_rng(3)
    v0, v1, v2 = rng.standard_normal((3, s.n))
    s.spmatvec(v0)                                   # leaves another product's sums behind
    want = [g.spmatvec(v) for v in (v1, v2)]
    d_v = [torch.from_numpy(v).cuda() for v in (v1, v2)]
    d_hv = [torch.zeros_like(x) for x in d_v]
    torch.cuda.synchronize()
    monkeypatch.setenv("NSS_WAIT_LIMIT", "0")
    got = [s.spmatvec(v) for v in (v1, v2)]
    for x, y in zip(d_v, d_hv):
        s.hv_device(x.data_ptr(), y.data_ptr())
    torch.cuda.synchronize()
    monkeypatch.delenv("NSS_WAIT_LIMIT")
    got += [y.cpu().numpy() for y in d_hv]
    # either path is a chain of at most 400 products: 800 roundings apart
    for x, w in zip(got, want + want):
        assert np.abs(x - w).max() <= 800 * 2.0 ** -53 * np.abs(w).max()
    assert np.abs(s.spmatvec(v1) - want[0]).max() <= 800 * 2.0 ** -53 * np.abs(want[0]).max()
    s.close()
    g.close()


@pytest.mark.parametrize("dr,kernels", [(4096, 5), (4097, 1)])
def test_the_largest_contracted_dimension(monkeypatch, dr, kernels):
    """The digit sums hold 4096 products; a wider sector keeps its superblock on
    the CUDA cores, also where the tensor cores are asked for."""
    import scipy.sparse as sp

    import nssdmrg_gb300 as nss
    nss.lib()
    monkeypatch.setenv("NSS_SPLIT64", "1")
    rng = np.random.default_rng(dr)
    s = nss.Superblock()
    d = rng.standard_normal(dr)
    s.upload([2], [dr], [0], [sp.csr_matrix(np.array([[1.5, 0.25], [0.25, -2.0]]))], [sp.diags(d).tocsr()], [], 0, 2, dr)
    v = rng.standard_normal(2 * dr)
    before = s.launches
    got = s.spmatvec(v).reshape(2, dr)
    assert s.launches - before == kernels
    w = v.reshape(2, dr)
    want = np.array([[1.5, 0.25], [0.25, -2.0]]) @ w + w * d
    mag = np.array([[1.5, 0.25], [0.25, 2.0]]) @ abs(w) + abs(w * d)
    assert (abs(got - want) <= 10 * 2.0 ** -53 * mag).all()
    s.close()
