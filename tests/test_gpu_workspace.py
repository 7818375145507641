"""The Lanczos workspace kept by a context from one size to the next.

Solves of different sizes, precisions and iteration caps one after the other
in one context: growing, shrinking within the kept block, beyond 64 MB (a cap
of 2 000 columns of 5 520 states is 88 MB) and back, where most of the block is
given back.  Every result is bit for bit that of a context of its own: the
arithmetic does not depend on where the arrays lie or what they held.  The tile
tuner is off: it would give the two contexts different plans of one class.
"""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


def _upload(nss, s, dims, seed):
    rng = np.random.default_rng(seed)
    sym = lambda d: sp.csr_matrix((lambda x: 0.5 * (x + x.T))(rng.standard_normal((d, d)) + 4 * np.diag(rng.standard_normal(d))))
    off = np.concatenate([[0], np.cumsum([a * b for a, b in dims])[:-1]]).astype(np.int64)
    s.upload([a for a, _ in dims], [b for _, b in dims], off, [sym(a) for a, _ in dims], [sym(b) for _, b in dims], [], 0,
             sum(a for a, _ in dims), sum(b for _, b in dims))


@pytest.mark.parametrize("budget", [0, 4 << 30])
def test_sizes_one_after_the_other(monkeypatch, budget):
    import nssdmrg_gb300 as nss
    monkeypatch.setenv("NSS_TC_AUTO", "0")
    nss.lib()
    small, mid, big = [(5, 7)], [(20, 30), (31, 17)], [(60, 70), (33, 40)]
    runs = [(small, 512, "NSS_PREC_FP64"), (mid, 512, "NSS_PREC_MIXED"), (big, 512, "NSS_PREC_FP64"),
            (mid, 512, "NSS_PREC_FP64"), (big, 2000, "NSS_PREC_FP64"), (small, 512, "NSS_PREC_MIXED"),
            (big, 512, "NSS_PREC_MIXED"), (small, 512, "NSS_PREC_FP64")]
    kept = nss.Superblock(0, hbm_budget=budget)
    for k, (dims, cap, precision) in enumerate(runs):
        own = nss.Superblock(0)
        out = []
        for s in (kept, own):
            _upload(nss, s, dims, k)
            ev, vec, num = s.sb_diag(neigen=1, nitermax=cap, tol=1e-12, precision=getattr(nss, precision))
            out.append((ev, vec, num))
        assert out[0][2] == out[1][2]
        assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
        own.close()
    kept.close()
