"""FP64 products on the tensor cores (k_sector_split.cu) against exact sums.

NSS_SPLIT64 forces the path at any size, so the edges of its tiles are
covered: sectors of 1, of 31 / 32 / 33, 63 / 64 / 65, 127 / 128 / 129 and 257
states (M = 128, N = 32 or 64, K in slabs of 64 read in groups of four),
vectors scaled by 2^-700 and 2^600, rows of very different size, constant and
all-ones operators (every digit sum of one sign), A with rounding-level rest
and with several sizeable entries, zero and non-finite elements.

Tolerance: the digit product errs by one rounding of each plane, the sum of
the planes and terms by one more each, and 2^-57 K max|H| max|W| per product:
3 * 2^-53 (|D_L| + |D_R| + |T|) + 2^-56 K (max|H| max|W|) per element, with the
exact value from integer arithmetic (Python's fractions through numpy longdouble
where it has 113 bits, else FP64 pairs).  The general FP64 chain is held to K 2^-53
sum |H||W| beside it.
"""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -53


def _two_sum(a, b):
    s = a + b
    t = s - a
    return s, (a - (s - t)) + (b - t)


def _split(a):
    c = 134217729.0 * a
    h = c - (c - a)
    return h, a - h


def _exact_matmul(A, B):
    """A @ B summed in FP64 pairs (Dekker products, compensated): 2^-100."""
    hi = np.zeros((A.shape[0], B.shape[1]))
    lo = np.zeros_like(hi)
    for k in range(A.shape[1]):
        a, b = A[:, k:k + 1], B[k:k + 1]
        p = a * b
        ah, al = _split(a)
        bh, bl = _split(b)
        e = ((ah * bh - p) + ah * bl + al * bh) + al * bl
        hi, r = _two_sum(hi, p)
        lo = lo + (r + e)
    return hi, lo


def _superblock(nss, dims, rng, make, term=None):
    """Sectors (dl, dr) with dense H from make(d); term: 'plain', 'rest', 'general'."""
    hl = [make(a) for a, _ in dims]
    hr = [make(b) for _, b in dims]
    off = np.concatenate([[0], np.cumsum([a * b for a, b in dims])[:-1]]).astype(np.int64)
    terms = []
    if term:
        for k, (a, b) in enumerate(dims):
            A = sp.diags(rng.choice([-1.0, 1.0], a)).tocsr()
            if term == "rest":
                A = (A + sp.csr_matrix(rng.standard_normal((a, a)) * 1e-17)).tocsr()
            if term == "general":
                A = (A + sp.csr_matrix(rng.standard_normal((a, a)) * (rng.random((a, a)) < 0.2))).tocsr()
            terms.append((0, k, k, 0, A, sp.diags(rng.standard_normal(b)).tocsr(), int(off[k]), int(off[k])))
    s = nss.Superblock()
    ml, mr = sum(a for a, _ in dims), sum(b for _, b in dims)
    s.upload([a for a, _ in dims], [b for _, b in dims], off, [sp.csr_matrix(h) for h in hl],
             [sp.csr_matrix(h) for h in hr], terms, 1 if term else 0, ml, mr)
    return s, hl, hr, off, {t[1]: t for t in terms}


def _check(s, dims, hl, hr, off, terms, v):
    got = s.spmatvec(v)
    for k, (a, b) in enumerate(dims):
        W = v[off[k]:off[k] + a * b].reshape(a, b)
        l, le = _exact_matmul(hl[k], W)
        r, re = _exact_matmul(W, hr[k].T.copy())
        t = np.zeros((a, b))
        if k in terms:
            A, B = terms[k][4], terms[k][5]
            t = np.asarray(A @ (B @ W.T).T)
        want = (l + r + t) + (le + re)
        mag = np.abs(l) + np.abs(r) + 4 * np.abs(t) + np.abs(want)
        cross = (a * np.abs(hl[k]).max() * np.abs(W).max(0, keepdims=True) +
                 b * np.abs(hr[k]).max() * np.abs(W).max(1, keepdims=True))
        tol = 3 * EPS * mag + 2.0 ** -56 * cross + (40 * EPS * (np.abs(A) @ (np.abs(B) @ np.abs(W.T)).T) if k in terms else 0)
        err = np.abs(got[off[k]:off[k] + a * b].reshape(a, b) - want)
        assert (err <= tol).all(), (k, a, b, float((err / np.maximum(tol, 1e-300)).max()))


@pytest.fixture()
def nss(monkeypatch):
    import nssdmrg_gb300 as nss
    nss.lib()
    monkeypatch.setenv("NSS_SPLIT64", "1")
    return nss


def _sym(rng, d):
    x = rng.standard_normal((d, d)) + 5.0 * np.diag(rng.standard_normal(d))
    return 0.5 * (x + x.T)


@pytest.mark.parametrize("dims", [
    [(1, 1)], [(1, 70), (33, 1)], [(31, 32), (32, 33), (63, 64), (64, 65)], [(127, 129), (128, 128), (129, 31)],
    [(257, 66), (5, 300)], [(200, 180)] * 3 + [(320, 330)],
], ids=str)
@pytest.mark.parametrize("term", [None, "plain", "rest", "general"])
def test_tiles_and_terms(nss, dims, term):
    rng = np.random.default_rng(sum(a * 7 + b for a, b in dims))
    s, hl, hr, off, terms = _superblock(nss, dims, rng, lambda d: _sym(rng, d), term)
    n = sum(a * b for a, b in dims)
    v = rng.standard_normal(n)
    _check(s, dims, hl, hr, off, terms, v)
    # rows and columns of very different size
    w = np.concatenate([(10.0 ** rng.uniform(-12, 0, (a, 1)) * rng.standard_normal((a, b)) *
                         10.0 ** rng.uniform(-6, 0, (1, b))).reshape(-1) for a, b in dims])
    _check(s, dims, hl, hr, off, terms, w)
    s.close()


@pytest.mark.parametrize("value", [1.0, -0.75, 1.0 / 3.0, 1.0 - 2.0 ** -53, 0.5 + 2.0 ** -30])
def test_digit_sums_of_one_sign(nss, value):
    """Constant operators and vectors: every partial sum at its largest."""
    dims = [(300, 290)]
    s, hl, hr, off, terms = _superblock(nss, dims, None, lambda d: np.full((d, d), value))
    _check(s, dims, hl, hr, off, terms, np.full(300 * 290, 1.0 - 2.0 ** -53))
    _check(s, dims, hl, hr, off, terms, np.full(300 * 290, value))
    s.close()


@pytest.mark.parametrize("scale", [2.0 ** -700, 2.0 ** 600, 2.0 ** -60])
def test_scaled_vectors(nss, scale):
    dims = [(70, 66), (40, 130)]
    rng = np.random.default_rng(5)
    s, hl, hr, off, terms = _superblock(nss, dims, rng, lambda d: _sym(rng, d), "rest")
    v = rng.standard_normal(70 * 66 + 40 * 130)
    np.testing.assert_array_equal(s.spmatvec(v * scale), s.spmatvec(v) * scale)   # a power of two changes no digit
    s.close()


def test_zero_and_non_finite(nss):
    dims = [(70, 66)]
    rng = np.random.default_rng(6)
    s, hl, hr, off, terms = _superblock(nss, dims, rng, lambda d: _sym(rng, d))
    v = rng.standard_normal(70 * 66)
    assert not s.spmatvec(0 * v).any()
    v[5 * 66 + 7] = np.nan
    got = s.spmatvec(v).reshape(70, 66)
    bad = np.zeros((70, 66), bool)
    bad[5] = True
    bad[:, 7] = True
    assert np.isnan(got[bad]).all() and np.isfinite(got[~bad]).all()
    s.close()
