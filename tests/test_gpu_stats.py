"""Kernel statistics of the FP64 loop in one kernel."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_plain_loop_counts_the_bytes_of_every_iteration(fe):
    rng = np.random.default_rng(5)
    n, levels = 20_011, (1500, 300, 50)
    feM = fe.AbstractFixedEffectSolver(
        [fe.FixedEffect.from_refs(rng.integers(1, m + 1, n), m) for m in levels], None, "CUDA",
        np.float64)
    feM.set_option(fe._lib.FE_OPT_PROFILE, 1)
    y, per = rng.standard_normal(n), []
    for tol in (1e-3, 1e-12):
        feM.reset_stats()
        feM.solve_residuals(y.copy(), tol=tol)
        stat = feM.kernel_stats()["plain_loop"]
        assert stat["launches"] == 1
        per.append(stat["bytes"] / feM.last_solve_info(1)["lsmr_iters"][0])
    feM.close()
    assert per[0] == pytest.approx(per[1], rel=1e-12)
    assert per[0] > n * (3 * 4 + 2 * 8)  # level ids of three effects, u read and written
