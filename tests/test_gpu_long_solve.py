"""Solves of thousands of iterations: a spectrum whose low end is dense.

The coefficients of several Ritz vectors then take more than the 48 KB of shared
memory that a kernel has without asking (ne x iterations > 6144).  H = H_L + H_R
has known eigenvalues, the sums of two lists; the energies have to meet them to
the tolerance, the residuals 3 tol |E|, and the vectors are orthogonal to 4e-15.
"""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


def _superblock(nss, low, high):
    rng = np.random.default_rng(2)
    ops = []
    for e in (low, high):
        q = np.linalg.qr(rng.standard_normal((len(e), len(e))))[0]
        x = (q * e) @ q.T
        ops.append(sp.csr_matrix(0.5 * (x + x.T)))
    s = nss.Superblock()
    s.upload([len(low)], [len(high)], [0], ops[:1], ops[1:], [], 0, len(low), len(high))
    return s, np.sort((low[:, None] + high[None]).reshape(-1))


@pytest.mark.parametrize("neigen", [1, 4])
def test_dense_low_end(neigen):
    import nssdmrg_gb300 as nss
    nss.lib()
    s, exact = _superblock(nss, -1 + 2 * np.linspace(0, 1, 65) ** 3, 0.05 * np.linspace(0, 1, 65) ** 2)
    ev, vec, products = s.sb_diag(neigen=neigen, tol=1e-12, nitermax=4000, seed=7)
    print(f"{neigen} states: {products} products, errors {np.abs(ev - exact[:neigen]).max():.1e}")
    assert products > 1536
    np.testing.assert_allclose(ev, exact[:neigen], rtol=0, atol=1e-12)
    for e in range(neigen):
        v = np.ascontiguousarray(vec[:, e])
        assert np.linalg.norm(s.spmatvec(v) - ev[e] * v) <= 3e-12 * abs(ev[0])
    assert np.abs(vec.T @ vec - np.eye(neigen)).max() <= 4e-15
    s.close()
