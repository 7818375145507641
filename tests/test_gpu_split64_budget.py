"""A context's memory budget and the tensor-core FP64 product.

The product's digits and planes take several times the operators' memory.  With
the smallest budget under which the superblock uploads and solves without them
(NSS_SPLIT64=0, found by bisection to 64 KiB), the same calls have to succeed
with them wanted (NSS_SPLIT64=1): the products then run on the CUDA cores.
"""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu

DIMS = [(120, 110), (90, 130), (64, 64)]


def _calls(nss, budget, steps, v):
    """The product and, from steps = 2 on, the lowest energy; None without memory."""
    rng = np.random.default_rng(8)
    off = np.concatenate([[0], np.cumsum([a * b for a, b in DIMS])[:-1]]).astype(np.int64)
    sym = lambda d: (lambda x: x + x.T)(rng.standard_normal((d, d)))
    hl, hr = [sp.csr_matrix(sym(a)) for a, _ in DIMS], [sp.csr_matrix(sym(b)) for _, b in DIMS]
    s = nss.Superblock(0, hbm_budget=budget)
    try:
        s.upload([a for a, _ in DIMS], [b for _, b in DIMS], off, hl, hr, [], 0, sum(a for a, _ in DIMS),
                 sum(b for _, b in DIMS))
        hv = s.spmatvec(v)
        ev = s.sb_diag(neigen=1, tol=1e-10, nitermax=300, want_vectors=False)[0][0] if steps > 1 else None
        return hv, ev, s.spmatvec(v)
    except nss.NssError as e:
        assert e.code == nss.NSS_ERR_NOMEM, str(e)
        return None
    finally:
        s.close()


@pytest.mark.parametrize("steps", [1, 2], ids=["product", "solve"])
def test_what_fitted_still_fits(monkeypatch, steps):
    import nssdmrg_gb300 as nss
    nss.lib()
    v = np.random.default_rng(9).standard_normal(sum(a * b for a, b in DIMS))
    monkeypatch.setenv("NSS_SPLIT64", "0")
    lo, hi = 0, 512 << 20
    want = _calls(nss, hi, steps, v)
    assert want is not None
    while hi - lo > 64 << 10:
        mid = (lo + hi) // 2
        lo, hi = (lo, mid) if _calls(nss, mid, steps, v) else (mid, hi)
    monkeypatch.setenv("NSS_SPLIT64", "1")
    for budget in (hi, hi + hi // 8, 2 * hi, 512 << 20):
        got = _calls(nss, budget, steps, v)
        assert got is not None, f"NSS_ERR_NOMEM with {budget} bytes where {hi} did"
        # chains of at most 250 products, or sums as exact
        for x in (got[0], got[2]):
            assert np.abs(x - want[0]).max() <= 500 * 2.0 ** -53 * np.abs(want[0]).max()
        if steps > 1:
            assert abs(got[1] - want[1]) <= 1e-10 * abs(want[1])
