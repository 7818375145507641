"""Partial reorthogonalisation against the tolerance and the vectors asked for.

An FP64 solve of 3072 states or more projects by estimate.  A basis of more
than 4096 columns projects at every step, so nitermax = 4200 gives the solve to
compare with.  The residual of a returned pair may exceed that solve's by what
the stopping test (tol |E|) and the estimates' threshold (half of tol, times
beta) allow: 3 tol |E| + 2 (its residual).  The vectors of several states are
orthogonal to the rounding of one projection: an inner product of two unit
vectors summed in FP64, below 4e-15.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [("MODEL_HEISENBERG_HALF", 10, 80), ("MODEL_HUBBARD", 4, 64)]
EVERY_STEP = 4200


@pytest.fixture(params=CASES, ids=lambda c: c[0])
def solver(request):
    import nssdmrg_gb300 as nss
    nss.lib()
    model, ldmrg, m = request.param
    kw = dict(u=4.0, hfmode=False, dmrg_qn=(0.5, 0.5)) if model == "MODEL_HUBBARD" else {}
    d = nss.DMRG(getattr(nss, model), ldmrg, m, lanc_neigen=1, **kw)
    d.prepare_last()
    assert d.sb.n > EVERY_STEP
    yield d.sb
    d.close()


def _residuals(s, ev, vec):
    return np.array([np.linalg.norm(s.spmatvec(np.ascontiguousarray(x)) - e * x) for e, x in zip(ev, vec.T)])


@pytest.mark.parametrize("neigen", [1, 3])
@pytest.mark.parametrize("tol", [1e-12, 1e-13, 1e-14, 0.0])
def test_residual_follows_the_tolerance(solver, tol, neigen):
    s, seeds = solver, (1234, 5)
    # the solves by estimate first: a context keeps a larger basis's workspace
    est = [s.sb_diag(neigen=neigen, tol=tol, seed=k) for k in seeds]
    for seed, (ev, vec, n_est) in zip(seeds, est):
        ref, rvec, n_all = s.sb_diag(neigen=neigen, tol=tol, seed=seed, nitermax=EVERY_STEP)
        res, rres = _residuals(s, ev, vec), _residuals(s, ref, rvec)
        print(f"N {s.n} states {neigen} tol {tol:g}: residuals / |E| {res / abs(ev[0])} ({n_est} products), "
              f"every step {rres / abs(ev[0])} ({n_all})")
        assert (res <= 3 * tol * abs(ev[0]) + 2 * rres).all()


@pytest.mark.parametrize("tol", [1e-12, 1e-14])
def test_vectors_of_several_states_are_orthogonal(solver, tol):
    s = solver
    ev, vec, _ = s.sb_diag(neigen=3, tol=tol)
    g = np.abs(vec.T @ vec - np.eye(3))
    print(f"N {s.n} tol {tol:g}: {g.max():.1e}")
    assert g.max() <= 4e-15
