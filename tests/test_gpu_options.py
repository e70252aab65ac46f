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


@pytest.mark.parametrize("T,kernel,options", [
    (np.float32, "coef_solve",
     [("EXPAND_VARIANT", 0), ("SEGSUM_VARIANT", 0), ("ROWSUM_VARIANT", 1),
      ("ABSORB", 0), ("ABSORB_SCALE", 0), ("FUSED_DEMEAN", 0), ("EXDM_PIPE", 0),
      ("FIRM_ATOMIC", 1), ("FUSED_RESID", 0), ("FUSED_RESID", 1), ("FUSED_RESID", 2)]),
    (np.float64, "plain_loop",
     [("EXPAND_VARIANT", 0), ("SEGSUM_VARIANT", 0), ("ROWSUM_VARIANT", 0)])])
def test_options_that_name_launched_kernels_select_them(fe, T, kernel, options):
    feM, y = _solver(fe, T)
    r0, _, _ = feM.solve_residuals(y.copy(), tol=1e-8)
    assert kernel in feM.kernel_stats()
    feM.close()
    for name, value in options:
        feM, _ = _solver(fe, T)
        feM.set_option(getattr(fe._lib, "FE_OPT_" + name), value)
        r, _, cv = feM.solve_residuals(y.copy(), tol=1e-8)
        assert cv and kernel not in feM.kernel_stats(), name
        feM.close()
        assert np.linalg.norm(r - r0) < 1e-6 * np.linalg.norm(r0)


@pytest.mark.parametrize("T", [np.float32, np.float64])
def test_graph_replay_of_the_launched_loops_matches_direct_launches(fe, T):
    out = []
    for graph in (1, 0):
        feM, y = _solver(fe, T)
        for name, value in (("PROFILE", 0), ("ROWSUM_VARIANT", 1), ("GRAPH", graph)):
            feM.set_option(getattr(fe._lib, "FE_OPT_" + name), value)
        out += [feM.solve_residuals(y.copy(), tol=1e-8) for _ in range(2)]
        feM.close()
    assert all(np.array_equal(r, out[0][0]) and it == out[0][1] for r, it, _ in out)
