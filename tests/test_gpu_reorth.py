"""Partial reorthogonalisation of the Lanczos basis.

The FP64 method projects at every step below 3072 states and by estimate
above; the FP32 phase projects by estimate until its basis fills an eighth of
the space.  Superblocks on both sides of those lines, solved to tol = 1e-12:
the solver stops at beta |s_m| <= tol |theta|, what the estimates let pass
adds at most their threshold (5e-13) times beta, and rounding 1e-16 ||H||
per step, so the residual of the returned vector stays below 3 tol |E|, and
the energy (its Rayleigh quotient) equals that of the other precision to
1e-12 |E|.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (model name, ldmrg, m): 70 to 67 072 states, 3072 between the third and fourth
CASES = [("MODEL_HEISENBERG_HALF", 4, 40), ("MODEL_HEISENBERG_HALF", 8, 40), ("MODEL_HEISENBERG_ONE", 5, 40),
         ("MODEL_HEISENBERG_HALF", 10, 64), ("MODEL_HUBBARD", 4, 64), ("MODEL_HUBBARD", 7, 256)]


@pytest.mark.parametrize("model,ldmrg,m", CASES)
def test_vectors_meet_the_residual_test(model, ldmrg, m):
    import nssdmrg_gb300 as nss
    nss.lib()
    kw = dict(u=4.0, hfmode=False, dmrg_qn=(0.5, 0.5)) if model == "MODEL_HUBBARD" else {}
    d = nss.DMRG(getattr(nss, model), ldmrg, m, lanc_neigen=1, **kw)
    d.prepare_last()
    s = d.sb
    energies = []
    for precision in (nss.NSS_PREC_FP64, nss.NSS_PREC_MIXED):
        for seed in (1234, 5):
            ev, vec, numop = s.sb_diag(neigen=1, tol=1e-12, seed=seed, precision=precision)
            v = np.ascontiguousarray(vec[:, 0])
            res = np.linalg.norm(s.spmatvec(v) - ev[0] * v)
            print(f"{model} N {s.n} precision {precision} seed {seed}: {numop} products, residual {res / abs(ev[0]):.1e} |E|")
            assert abs(np.linalg.norm(v) - 1.0) <= 1e-14 * np.sqrt(s.n)
            assert res <= 3e-12 * abs(ev[0])
            energies.append(ev[0])
    d.close()
    assert max(energies) - min(energies) <= 1e-12 * abs(energies[0])
