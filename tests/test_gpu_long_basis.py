"""A Krylov basis of more than 4096 columns (nitermax) has no room for the
estimates of the partial reorthogonalisation and projects at every step.
Solved to tol = 1e-12 the residual stays below 3 tol |E|, and the energy, a
Rayleigh quotient, agrees with that of a short basis to 1e-12 |E|.
"""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


def _superblock(nss, dims, reps, several, rng):
    def sym(d):
        x = rng.standard_normal((d, d)) / np.sqrt(d) + 2.0 * np.diag(rng.standard_normal(d))
        return sp.csr_matrix(0.5 * (x + x.T))

    def partial(rows, cols):
        n = min(rows, cols)
        r, c = rng.permutation(rows)[:n], rng.permutation(cols)[:n]
        m = sp.csr_matrix((rng.uniform(0.3, 1.0, n) * rng.choice([-1.0, 1.0], n), (r, c)), shape=(rows, cols))
        if several:
            m = sp.csr_matrix(m + sp.csr_matrix(0.3 * rng.standard_normal((rows, cols)) * (rng.random((rows, cols)) < 2.0 / cols)))
        return m

    off = np.concatenate([[0], np.cumsum([a * b for a, b in dims])[:-1]]).astype(np.int64)
    terms = []
    for k in range(len(dims) - 1):
        (a0, b0), (a1, b1) = dims[k], dims[k + 1]
        for t in range(reps):
            A, B = partial(a1, a0), partial(b1, b0)
            terms.append((2 * t, k + 1, k, 0, A, B, int(off[k + 1]), int(off[k])))
            terms.append((2 * t + 1, k, k + 1, 0, A.T.tocsr(), B.T.tocsr(), int(off[k]), int(off[k + 1])))
    s = nss.Superblock()
    s.upload([a for a, _ in dims], [b for _, b in dims], off, [sym(a) for a, _ in dims], [sym(b) for _, b in dims],
             terms, 2 * reps, sum(a for a, _ in dims), sum(b for _, b in dims))
    return s


def _residual(s, ev, vec):
    v = np.ascontiguousarray(vec[:, 0])
    return np.linalg.norm(s.spmatvec(v) - ev[0] * v) / abs(ev[0])


@pytest.mark.parametrize("precision", ["NSS_PREC_FP64", "NSS_PREC_MIXED"])
def test_long_krylov_basis(precision):
    import nssdmrg_gb300 as nss
    nss.lib()
    s = _superblock(nss, [(60, 70), (33, 40)], 1, False, np.random.default_rng(3))
    ev, vec, _ = s.sb_diag(neigen=1, tol=1e-12)
    ev2, vec2, _ = s.sb_diag(neigen=1, nitermax=5000, tol=1e-12, precision=getattr(nss, precision))
    assert _residual(s, ev2, vec2) <= 3e-12
    assert abs(ev[0] - ev2[0]) <= 1e-12 * abs(ev[0])
    s.close()


def test_long_krylov_basis_batch():
    import nssdmrg_gb300 as nss
    nss.lib()
    sbs = [_superblock(nss, [(60, 70), (33, 40)], 1, False, np.random.default_rng(k)) for k in (3, 4)]
    want = [s.sb_diag(neigen=1, tol=1e-12)[0][0] for s in sbs]
    got, _ = nss.eigh_batch(sbs, nitermax=5000, tol=1e-12)
    for w, g in zip(want, got):
        assert abs(w - g) <= 1e-12 * abs(w)
    for s in sbs:
        s.close()
