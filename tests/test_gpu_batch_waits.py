"""A batch whose FP64 product on the tensor cores gives up a wait.

NSS_WAIT_LIMIT=0 (a test knob) makes every bounded wait of k_sector_split run
out: the kernel returns without its sums.  nss_batch_step must report that, and
the next batch on the context is right.
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


def test_batch_reports_a_product_that_gave_up(monkeypatch):
    """With a loose tolerance the FP32 phase is the whole solve and the batch's
    last step is one FP64 product; the same steps again with that product's
    waits at zero have to end in an error, and the next batch is right."""
    nss, s, ref = _upload(monkeypatch, "1")

    def steps(limit_at):
        eng = nss.BatchEngine(s)
        eng.add(s, seed=1, tol=1e-5)
        done, n = [], 0
        try:
            while eng.inflight and n < 200:
                n += 1
                if n == limit_at:
                    monkeypatch.setenv("NSS_WAIT_LIMIT", "0")
                done += eng.step()
        finally:
            monkeypatch.delenv("NSS_WAIT_LIMIT", raising=False)
            eng.close()
        return n, done

    n, done = steps(0)
    assert len(done) == 1 and abs(done[0][1] - ref) <= 1e-6 * abs(ref)
    s.spmatvec(np.random.default_rng(4).standard_normal(s.n))
    with pytest.raises(nss.NssError) as ei:
        steps(n)
    assert ei.value.code == nss.NSS_ERR_CUDA and "timed out" in str(ei.value), str(ei.value)
    n2, done = steps(0)
    assert n2 == n and len(done) == 1 and abs(done[0][1] - ref) <= 1e-6 * abs(ref)
    s.close()
