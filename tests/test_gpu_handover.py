"""Columns that the coefficient side cannot finish: the tile goes on from where
it stands instead of being solved again, and columns with a large mean stay.

The bar is the repository's 1e-6 on the residual's relative 2-norm (relative
to the column where the fit is exact).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

REL = 1e-6
N = 20_011


def _problem(fe, nlev, weighted=False, interacted=False, seed=5):
    rng = np.random.default_rng(seed)
    refs = [rng.integers(1, m + 1, N) for m in nlev]
    inter = [None] * len(nlev)
    if interacted:
        inter[0] = rng.uniform(0.5, 1.5, N)
    w = rng.uniform(0.5, 1.5, N) if weighted else None
    feM = fe.AbstractFixedEffectSolver(
        [fe.FixedEffect.from_refs(r, m, a) for r, m, a in zip(refs, nlev, inter)], w, "CUDA",
        np.float32)
    feM.set_option(fe._lib.FE_OPT_PROFILE, 1)
    return feM, refs, inter, w, rng


def _oracle(oracle, Y, refs, nlev, inter, w):
    return oracle.solve_residuals_cols(Y.astype(np.float64), refs, list(nlev), inter, w,
                                       tol=1e-10)[0]


def _exact(refs, nlev, inter, rng):
    return sum(rng.standard_normal(m + 1)[r] * (1.0 if a is None else a)
               for r, m, a in zip(refs, nlev, inter))


@pytest.mark.parametrize("nlev", [(1500, 300), (1500, 300, 50), (1500, 300, 50, 7)])
@pytest.mark.parametrize("weighted,interacted", [(False, False), (True, False), (True, True)])
@pytest.mark.parametrize("cols", [1, 3, 8])
def test_exact_columns_are_finished_from_the_coefficients(fe, oracle, nlev, weighted, interacted,
                                                          cols):
    feM, refs, inter, w, rng = _problem(fe, nlev, weighted, interacted)
    Y = rng.standard_normal((N, cols)) + (refs[0] % 7)[:, None] * 0.4
    Y[:, cols // 2] = _exact(refs, nlev, inter, rng)
    Y = np.asfortranarray(Y.astype(np.float32))
    R, its, cv = feM.solve_residuals(Y.copy(order="F"), tol=1e-8)
    stats = feM.kernel_stats()
    feM.close()
    assert "coef_solve" in stats and "demean64" in stats
    assert "expand" not in stats  # no iteration on the row side
    R_o = _oracle(oracle, Y, refs, nlev, inter, w)
    assert cv.all() and its.max() < 60
    for j in range(cols):
        of = Y[:, j] if j == cols // 2 else R_o[:, j]
        assert np.linalg.norm(R[:, j] - R_o[:, j]) < REL * np.linalg.norm(of)


@pytest.mark.parametrize("weighted,interacted", [(False, False), (True, False), (True, True)])
@pytest.mark.parametrize("cols", [1, 8])
@pytest.mark.parametrize("mean", [1e2, 1e5])
def test_columns_with_a_large_mean_stay(fe, oracle, weighted, interacted, cols, mean):
    nlev = (1500, 300, 50)
    feM, refs, inter, w, rng = _problem(fe, nlev, weighted, interacted)
    Y = rng.standard_normal((N, cols))
    big = mean if inter[0] is None else mean * inter[0]
    Y[:, 0] += big
    Y = np.asfortranarray(Y.astype(np.float32))
    R, _, cv = feM.solve_residuals(Y.copy(order="F"), tol=1e-8)
    stats = feM.kernel_stats()
    feM.close()
    assert "coef_solve" in stats and "demean64" not in stats
    R_o = _oracle(oracle, Y, refs, nlev, inter, w)
    assert cv.all()
    for j in range(cols):
        assert np.linalg.norm(R[:, j] - R_o[:, j]) < REL * np.linalg.norm(R_o[:, j])


@pytest.mark.parametrize("cols", [1, 5])
def test_a_column_constant_within_levels_is_handed_over_at_once(fe, oracle, cols):
    # what is left of it is rounding, on which LSMR iterates as it does on the
    # row side (and as the reference does)
    nlev = (1500, 300, 50)
    feM, refs, inter, w, rng = _problem(fe, nlev)
    Y = rng.standard_normal((N, cols))
    Y[:, 0] = rng.standard_normal(nlev[0] + 1)[refs[0]]
    Y = np.asfortranarray(Y.astype(np.float32))
    R, its, cv = feM.solve_residuals(Y.copy(order="F"), tol=1e-8)
    feM.set_option(fe._lib.FE_OPT_EXPAND_VARIANT, 0)
    feM.set_option(fe._lib.FE_OPT_SEGSUM_VARIANT, 0)
    R1, its1, cv1 = feM.solve_residuals(Y.copy(order="F"), tol=1e-8)
    feM.close()
    assert np.array_equal(cv, cv1) and cv[1:].all()
    assert np.abs(R[:, 0]).max() < 1e-12
    R_o = _oracle(oracle, Y, refs, nlev, inter, w)
    for j in range(1, cols):
        assert np.linalg.norm(R[:, j] - R_o[:, j]) < REL * np.linalg.norm(R_o[:, j])


def test_a_tolerance_out_of_reach(fe, oracle):
    # no round can meet tol = 0: reported as not converged, and not for long
    nlev = (1500, 300, 50)
    feM, refs, inter, w, rng = _problem(fe, nlev)
    Y = np.asfortranarray(rng.standard_normal((N, 2)).astype(np.float32))
    R, its, cv = feM.solve_residuals(Y.copy(order="F"), tol=0.0)
    feM.close()
    R_o = _oracle(oracle, Y, refs, nlev, inter, w)
    assert not cv.any() and its.max() < 200
    for j in range(2):
        assert np.linalg.norm(R[:, j] - R_o[:, j]) < REL * np.linalg.norm(R_o[:, j])


def test_nan_and_zero_columns_beside_an_exact_one(fe, oracle):
    nlev = (1500, 300, 50)
    feM, refs, inter, w, rng = _problem(fe, nlev)
    Y = rng.standard_normal((N, 4))
    Y[:, 1] = 0.0
    Y[7, 2] = np.nan
    Y[:, 3] = _exact(refs, nlev, inter, rng)
    Y = np.asfortranarray(Y.astype(np.float32))
    R, its, cv = feM.solve_residuals(Y.copy(order="F"), tol=1e-8)
    feM.close()
    assert list(cv) == [True, True, False, True] and its[2] <= 2
    assert not R[:, 1].any() and np.isnan(R[7, 2])
    r_o = _oracle(oracle, Y[:, :1], refs, nlev, inter, w)[:, 0]
    assert np.linalg.norm(R[:, 0] - r_o) < REL * np.linalg.norm(r_o)
    assert np.linalg.norm(R[:, 3]) < REL * np.linalg.norm(Y[:, 3])
