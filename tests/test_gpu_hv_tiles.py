"""The FP64 product's warp tiles (k_hv_fp64): 4 x 8 outputs, K in slabs of 32.

Sectors at the edges of the tiles and slabs; A x B terms of one entry a row
(four in flight), rows of A with several entries (16 a round) and rows of B with
several; and enough tiles (4 800, the grid holds 3 040) that warps take their
next one from the queue, twice in a row, since a launch has to leave the queue
as it found it.  NSS_SPLIT64=0 keeps the products on this kernel.

Tolerance: an output is a chain of K fused additions and so is the reference's:
2 (K + 2) 2^-53 sum |a||b| with K the number of products of the output.
"""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -53


@pytest.mark.parametrize("kind", ["none", "single", "rows of A", "rows of B"])
@pytest.mark.parametrize("dims", [
    [(1, 1)], [(3, 7), (4, 8), (5, 9), (1, 33)], [(31, 33), (32, 32), (33, 31), (64, 65)], [(60, 60)] * 40,
], ids=lambda d: f"{len(d)}x{d[0]}")
def test_product(monkeypatch, dims, kind):
    import nssdmrg_gb300 as nss
    nss.lib()
    monkeypatch.setenv("NSS_SPLIT64", "0")
    rng = np.random.default_rng(len(dims) + dims[0][0])
    dense = lambda d: rng.standard_normal((d, d))
    hl, hr = [dense(a) for a, _ in dims], [dense(b) for _, b in dims]
    off = np.concatenate([[0], np.cumsum([a * b for a, b in dims])[:-1]]).astype(np.int64)
    terms, mats = [], {}
    for k, (a1, b1) in enumerate(dims if kind != "none" else []):
        for t in range(5):                           # one more than are in flight
            q = (k + t) % len(dims)
            a0, b0 = dims[q]
            A = sp.csr_matrix((rng.standard_normal(a1), (np.arange(a1), rng.integers(0, a0, a1))), shape=(a1, a0))
            B = sp.csr_matrix((rng.choice([-1.0, 1.0], b1) if t % 2 else rng.standard_normal(b1),
                               (np.arange(b1), rng.integers(0, b0, b1))), shape=(b1, b0))
            if kind == "rows of A" and t != 1:
                A = sp.csr_matrix(rng.standard_normal((a1, a0)) * (rng.random((a1, a0)) < 0.6))
            if kind == "rows of B" and t == 2:
                B = sp.csr_matrix(rng.standard_normal((b1, b0)) * (rng.random((b1, b0)) < 0.3))
            terms.append((t, k, q, 0, A, B, int(off[k]), int(off[q])))
            mats.setdefault(k, []).append((q, A, B))
    s = nss.Superblock()
    s.upload([a for a, _ in dims], [b for _, b in dims], off, [sp.csr_matrix(h) for h in hl],
             [sp.csr_matrix(h) for h in hr], terms, 5 if terms else 0, sum(a for a, _ in dims), sum(b for _, b in dims))
    v = rng.standard_normal(s.n)
    W = [v[o:o + a * b].reshape(a, b) for o, (a, b) in zip(off, dims)]
    for _ in range(2):
        got = s.spmatvec(v)
        for k, (a, b) in enumerate(dims):
            want, mag, n = hl[k] @ W[k] + W[k] @ hr[k].T, abs(hl[k]) @ abs(W[k]) + abs(W[k]) @ abs(hr[k].T), a + b
            for q, A, B in mats.get(k, []):
                want = want + (B @ (A @ W[q]).T).T
                mag = mag + (abs(B) @ (abs(A) @ abs(W[q])).T).T
                n += 2 * int(np.diff(A.indptr).max()) * int(np.diff(B.indptr).max())
            err = np.abs(got[off[k]:off[k] + a * b].reshape(a, b) - want)
            assert (err <= 2 * (n + 2) * EPS * mag).all(), (k, a, b, float((err / mag).max()))
    s.close()
