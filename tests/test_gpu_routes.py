"""Which narrow solves run in one kernel: shapes on both sides of the measured
lines.  Those on the launched side were slower in one kernel."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _route(fe, T, n, levels, cols, weighted, interacted):
    rng = np.random.default_rng(1)
    fes = [fe.FixedEffect.from_refs(rng.integers(1, m + 1, n), m,
                                    rng.uniform(0.5, 1.5, n) if interacted and k == len(levels) - 1
                                    else None) for k, m in enumerate(levels)]
    feM = fe.AbstractFixedEffectSolver(fes, rng.uniform(0.5, 1.5, n) if weighted else None, "CUDA", T)
    feM.set_option(fe._lib.FE_OPT_PROFILE, 1)
    feM.solve_residuals(np.asfortranarray(rng.standard_normal((n, cols)).astype(T)), tol=1e-8,
                        maxiter=6)
    stats = feM.kernel_stats()
    feM.close()
    return "coef_solve" in stats or "plain_loop" in stats


# mixed precision: levels of two rows with many elements, interacted effects
@pytest.mark.parametrize("n,levels,cols,weighted,interacted,one", [
    (3_000_000, (1_500_000, 600_000), 8, False, False, False),
    (3_000_000, (300_000, 150_000), 8, False, False, True),
    (3_000_000, (1_500_000, 600_000), 1, True, False, True),
    (3_000_000, (300_000, 1000, 30), 1, True, True, True),
    (3_000_000, (300_000, 150_000, 75_000), 1, True, True, False),
    (1_000_000, (100_000, 1000, 30), 2, True, True, False),
    (1_000_000, (100_000, 1000, 30), 4, True, True, True),
    (1_000_000, (100_000, 50_000, 25_000, 12_500), 1, True, True, False),
    (1_000_000, (100_000, 50_000, 25_000, 12_500), 1, False, False, True),
    # the row side's inner solves stall on these
    (1_000_000, (500_000, 200_000, 50_000, 10_000), 1, True, True, True),
    (2_000_000, (1_000_000, 500_000, 100_000), 2, True, True, True)])
def test_mixed_solves(fe, n, levels, cols, weighted, interacted, one):
    assert _route(fe, np.float32, n, levels, cols, weighted, interacted) == one


@pytest.mark.parametrize("n,levels,cols,weighted,interacted,one", [
    (2_400_000, (240_000, 30), 1, False, False, True),
    (2_400_000, (240_000, 30), 1, True, True, False),
    (300_000, (15_000, 500, 20, 6), 8, False, False, False),
    (300_000, (30_000, 15_000, 7500, 3750), 8, False, False, True),
    (300_000, (30_000, 15_000, 7500, 3750), 8, True, False, False),
    (100_000, (10_000, 30, 10), 4, False, False, False),
    (300_000, (30_000, 30, 10), 4, False, False, True),
    (100_000, (10_000, 5000, 2500), 4, True, True, False)])
def test_fp64_solves(fe, n, levels, cols, weighted, interacted, one):
    assert _route(fe, np.float64, n, levels, cols, weighted, interacted) == one
