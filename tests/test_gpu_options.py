"""Plan options on the calls that the one-kernel solves take by default."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N, LEVELS = 20_011, (1500, 300, 50)


def _solver(fe, T):
    rng = np.random.default_rng(5)
    feM = fe.AbstractFixedEffectSolver(
        [fe.FixedEffect.from_refs(rng.integers(1, m + 1, N), m) for m in LEVELS], None, "CUDA", T)
    feM.set_option(fe._lib.FE_OPT_PROFILE, 1)
    return feM, rng.standard_normal(N).astype(T)


def test_inner_rho_ends_the_inner_solves_of_the_coefficient_side(fe):
    # the default needs one inner solve for 1e-10; a drop of 1e-3 each needs
    # at least three, and gives the same residual
    feM, y = _solver(fe, np.float32)
    r0, _, cv0 = feM.solve_residuals(y.copy(), tol=1e-10)
    assert cv0 and feM.last_solve_info(1)["rounds"][0] == 1
    feM.set_option(fe._lib.FE_OPT_INNER_RHO, 1e-3)
    r, _, cv = feM.solve_residuals(y.copy(), tol=1e-10)
    assert cv and feM.last_solve_info(1)["rounds"][0] >= 3
    assert "coef_solve" in feM.kernel_stats()
    feM.close()
    assert np.linalg.norm(r - r0) < 1e-6 * np.linalg.norm(r0)
