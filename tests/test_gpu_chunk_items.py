"""The persistent kernel's products (hv32_item) at the edges of its tiles.

Sectors of 1 to 257 states: both products staged together up to 48, in parts
above, the K range in rounds above 128; tiles of 32; A x B tables of one
element a row (four gathered ahead, sixteen staged at once) and rows of several
elements (the general loop).  A chain of couplings between the sectors spreads
the ground state over all of them, so a wrong element of any sector's product
keeps the mixed method's refinement from converging: it would be counted as a
fallback to FP64.  Solved to tol = 1e-12, so the residual stays below
3 tol |E| (what the estimates of the reorthogonalisation let pass, and
rounding, add less than tol), and the energy, a Rayleigh quotient, agrees with
the FP64 method's to 1e-12 |E|.
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


@pytest.mark.parametrize("several", [False, True])
@pytest.mark.parametrize("reps", [1, 3, 9])
@pytest.mark.parametrize("dims", [
    [(1, 1), (3, 40), (31, 48), (33, 47)], [(48, 49), (49, 33), (64, 65), (65, 64)],
    [(127, 128), (128, 129), (129, 130), (40, 257)], [(97, 5), (2, 161), (32, 32)],
], ids=str)
def test_every_sector_enters_the_ground_state(dims, reps, several):
    import nssdmrg_gb300 as nss
    nss.lib()
    s = _superblock(nss, dims, reps, several, np.random.default_rng(sum(3 * a + b for a, b in dims) + reps))
    ev64, _, n64 = s.sb_diag(neigen=1, nitermax=1000, tol=1e-12)
    ev, vec, num = s.sb_diag(neigen=1, nitermax=1000, tol=1e-12, precision=nss.NSS_PREC_MIXED)
    res = _residual(s, ev, vec)
    print(f"N {s.n}: {n64} products FP64, {num} mixed, {s.refine_stats()}, residual {res:.1e} |E|")
    assert s.refine_stats()[2] == 0
    assert res <= 3e-12
    assert abs(ev[0] - ev64[0]) <= 1e-12 * abs(ev64[0])
    s.close()
