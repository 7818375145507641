"""FP64 products on the tensor cores, element by element.

The digits of an operand are relative to the largest element of its row, so
operands with elements of very different size, or products that meet in small
elements only, are where a product through them could have fewer bits than one
summed in FP64.  nss_hv promises an FP64 chain's error for every element:
(Dl + Dr + terms + 8) 2^-53 (|H_L||W| + |W||H_R^T| + |A||W||B^T|), and beside
it 2^-1074 per operation where results leave the normal range.  The reference
sums in FP64 pairs.
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


def _matmul(A, B):
    """A @ B in FP64 pairs (Dekker products, compensated sums)."""
    hi, lo = np.zeros((A.shape[0], B.shape[1])), np.zeros((A.shape[0], B.shape[1]))
    for k in range(A.shape[1]):
        a, b = A[:, k:k + 1], B[k:k + 1]
        p = a * b
        (ah, al), (bh, bl) = _split(a), _split(b)
        hi, r = _two_sum(hi, p)
        lo += r + (((ah * bh - p) + ah * bl + al * bh) + al * bl)
    return hi + lo


class _Sb:
    """Sectors (dl, dr) with given dense H and terms (out, in, A, B)."""

    def __init__(self, monkeypatch, dims, hl, hr, terms=(), split="1", **kw):
        import nssdmrg_gb300 as nss
        nss.lib()
        monkeypatch.setenv("NSS_SPLIT64", split)
        self.dims, self.hl, self.hr, self.terms = dims, hl, hr, list(terms)
        self.off = np.concatenate([[0], np.cumsum([a * b for a, b in dims])[:-1]]).astype(np.int64)
        self.s = nss.Superblock(0, **kw)
        up = [(t, k, q, 0, sp.csr_matrix(A), sp.csr_matrix(B), int(self.off[k]), int(self.off[q]))
              for t, (k, q, A, B) in enumerate(self.terms)]
        self.s.upload([a for a, _ in dims], [b for _, b in dims], self.off, [sp.csr_matrix(h) for h in hl],
                      [sp.csr_matrix(h) for h in hr], up, len(up), sum(a for a, _ in dims), sum(b for _, b in dims))
        self.n = sum(a * b for a, b in dims)

    def sectors(self, v):
        return [v[o:o + a * b].reshape(a, b) for o, (a, b) in zip(self.off, self.dims)]

    def check(self, v, scale=1.0):
        """The product of v * scale (a power of two) against the exact one of v."""
        got = self.sectors(self.s.spmatvec(v * scale))
        W = self.sectors(v)
        for k, (a, b) in enumerate(self.dims):
            parts = [(_matmul(self.hl[k], W[k]), abs(self.hl[k]) @ abs(W[k]), a),
                     (_matmul(W[k], self.hr[k].T.copy()), abs(W[k]) @ abs(self.hr[k].T), b)]
            for ko, q, A, B in self.terms:
                if ko == k:
                    parts.append((_matmul(_matmul(A, W[q]), B.T.copy()), abs(A) @ abs(W[q]) @ abs(B.T),
                                  int((A != 0).sum(1).max()) + int((B != 0).sum(1).max())))
            want = sum(p[0] for p in parts)
            mag = sum(p[1] for p in parts)
            ops = sum(p[2] for p in parts) + 8
            tol = ops * (EPS * mag * scale + 2.0 ** -1074)
            err = np.abs(got[k] - want * scale)
            assert (err <= tol).all(), (k, a, b, float((err / np.maximum(tol, 1e-300)).max()))


DIMS = [[(70, 66), (40, 130)], [(200, 180), (33, 5), (1, 300)]]


def _operators(kind, dims, rng):
    def make(d):
        if kind == "diagonal":
            return np.diag(rng.standard_normal(d))
        if kind == "near diagonal":
            return np.diag(rng.standard_normal(d)) + 1e-11 * rng.standard_normal((d, d))
        if kind == "graded":
            i = np.arange(d)
            return rng.standard_normal((d, d)) * 10.0 ** (-8.0 * abs(i[:, None] - i) / d)
        if kind == "sparse":
            return rng.standard_normal((d, d)) * (rng.random((d, d)) < 3.0 / d)
        return rng.standard_normal((d, d))
    return [make(a) for a, _ in dims], [make(b) for _, b in dims]


def _vector(kind, dims, rng):
    out = []
    for a, b in dims:
        w = rng.standard_normal((a, b))
        i, j = np.arange(a)[:, None] / a, np.arange(b)[None] / b
        if kind == "graded":
            w = w * 10.0 ** (-6.0 * (i + j))
        if kind == "steep":
            w = w * 10.0 ** (-20.0 * abs(i - j))
        if kind == "one element":
            w = np.zeros((a, b))
            w[a // 2, b // 3] = 0.7
        out.append(w.reshape(-1))
    return np.concatenate(out)


@pytest.mark.parametrize("vector", ["normal", "graded", "steep", "one element"])
@pytest.mark.parametrize("operators", ["diagonal", "near diagonal", "graded", "sparse", "dense"])
@pytest.mark.parametrize("dims", DIMS, ids=["two", "three"])
def test_every_element_as_a_chain(monkeypatch, dims, operators, vector):
    rng = np.random.default_rng(len(operators) * 10 + len(vector))
    sb = _Sb(monkeypatch, dims, *_operators(operators, dims, rng))
    v = _vector(vector, dims, rng)
    sb.check(v)
    sb.check(v)                                      # the product leaves its scratch as it found it
    sb.s.close()


def _cross(dims, rng, small):
    """Terms between sectors: +-1 in a shifted diagonal, `small` beside it in half of A."""
    out = []
    for k, (a1, b1) in enumerate(dims):
        q = (k + 1) % len(dims)
        a0, b0 = dims[q]
        A = np.zeros((a1, a0))
        A[np.arange(a1), np.arange(a1) % a0] = rng.choice([-1.0, 1.0], a1)
        rest = small * rng.standard_normal((a1, a0)) * (rng.random((a1, a0)) < 0.5)
        A = np.where(A != 0, A, rest)
        B = np.zeros((b1, b0))
        B[np.arange(b1), rng.integers(0, b0, b1)] = rng.standard_normal(b1)
        out.append((k, q, A, B))
    return out


@pytest.mark.parametrize("small", [1e-13, 1e-17])
def test_small_entries_of_a_alone(monkeypatch, small):
    """Rows of A whose large entry meets a zero row of the vector, so that only
    the small entries count; and rows where it meets a tiny one."""
    dims = [(70, 66), (40, 130), (90, 33)]
    rng = np.random.default_rng(11)
    zeros = [np.zeros((a, a)) for a, _ in dims], [np.zeros((b, b)) for _, b in dims]
    sb = _Sb(monkeypatch, dims, *zeros, _cross(dims, rng, small))
    for tiny in (0.0, 1e-18):
        v = rng.standard_normal(sb.n)
        for w in sb.sectors(v):
            w[::2] *= tiny
        sb.check(v)
    v = _vector("steep", dims, rng)
    sb.check(v)
    sb.s.close()


@pytest.mark.parametrize("scale", [2.0 ** -1030, 2.0 ** -1050, 2.0 ** -1070])
def test_results_below_the_normal_range(monkeypatch, scale):
    dims = [(70, 66), (40, 130)]
    rng = np.random.default_rng(12)
    sb = _Sb(monkeypatch, dims, *_operators("dense", dims, rng))
    v = np.round(rng.standard_normal(sb.n), 0)       # a few bits, so that v * scale is exact
    sb.check(v, scale)
    sb.s.close()


def test_small_products_of_normal_operands(monkeypatch):
    """Operators and a vector in the normal range whose products lie below it."""
    dims = [(70, 66), (40, 130)]
    rng = np.random.default_rng(15)
    hl, hr = ([np.round(h) * 2.0 ** -60 for h in x] for x in _operators("dense", dims, rng))
    sb = _Sb(monkeypatch, dims, hl, hr)
    v = np.round(rng.standard_normal(sb.n), 0)
    for scale in (2.0 ** -962, 2.0 ** -985, 2.0 ** -1010):
        sb.check(v, scale)
    sb.s.close()


@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
def test_non_finite_elements_as_a_chain(monkeypatch, value):
    """The elements an Inf or NaN reaches, and how, are those of the FP64 chain;
    the others keep their value."""
    dims = [(70, 66), (40, 130), (90, 33)]
    rng = np.random.default_rng(13)
    hl, hr = _operators("dense", dims, rng)
    hl[0][:, 5] = 0.0                                # 0 x Inf
    terms = _cross(dims, rng, 1e-15)
    v = rng.standard_normal(sum(a * b for a, b in dims))
    # in columns that the terms of sectors 2 and 0 read
    cols = [int(np.nonzero(terms[k][3])[1][3]) for k in (2, 0)]
    a, b = _Sb(monkeypatch, dims, hl, hr, terms), _Sb(monkeypatch, dims, hl, hr, terms, split="0")
    for at in (5 * 66 + cols[0], 70 * 66 + 3 * 130 + cols[1]):
        w = v.copy()
        w[at] = value
        got, want = a.s.spmatvec(w), b.s.spmatvec(w)
        np.testing.assert_array_equal(np.isnan(got), np.isnan(want))
        inf = np.isinf(want)
        np.testing.assert_array_equal(np.isinf(got), inf)
        np.testing.assert_array_equal(got[inf], want[inf])
        fin = np.isfinite(want)
        assert 0 < fin.sum() < fin.size
        # both are chains of at most 300 operations on elements of order one
        np.testing.assert_allclose(got[fin], want[fin], rtol=0, atol=600 * EPS * 300)
    a.s.close()
    b.s.close()


def test_a_non_finite_row_among_small_entries(monkeypatch):
    """An Inf or NaN that the small entries of A reach goes to its own column
    alone; the other columns keep what the small entries give."""
    dims = [(70, 66), (40, 130), (90, 33)]
    rng = np.random.default_rng(14)
    zeros = [np.zeros((a, a)) for a, _ in dims], [np.zeros((b, b)) for _, b in dims]
    terms = _cross(dims, rng, 1e-14)
    col = int(np.nonzero(terms[2][3])[1][3])
    sb, ref = _Sb(monkeypatch, dims, *zeros, terms), _Sb(monkeypatch, dims, *zeros, terms, split="0")
    v = rng.standard_normal(sb.n)
    w = sb.sectors(v)[0]
    w[::2] = 0.0                                     # sector 2's large entries of A meet zeros
    for value in (np.nan, np.inf):
        w[6, col] = value
        got, want = sb.s.spmatvec(v), ref.s.spmatvec(v)
        np.testing.assert_array_equal(np.isnan(got), np.isnan(want))
        fin = np.isfinite(want)
        np.testing.assert_array_equal(np.isfinite(got), fin)
        # chains of at most 70 products
        np.testing.assert_allclose(got[fin], want[fin], rtol=200 * EPS, atol=200 * EPS * 1e-14 * 30)
        sub = sb.sectors(want)[2][::2]
        assert not np.isfinite(sub).all() and 0 < np.abs(sub[np.isfinite(sub)]).max() < 1e-10
    sb.s.close()
    ref.s.close()
