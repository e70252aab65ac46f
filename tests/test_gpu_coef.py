"""The coefficient-side solve (FP32 columns, mixed precision, tiles of up to 8
columns) against the oracle, at the sizes where its work items change: levels
of a window and longer, levels of several pieces, empty levels, every tile
width, number of fixed effects and kind of weight.

The bar is the repository's 1e-6 on the residual's relative 2-norm: the FP64
test at 1e-8 and the rounding of the returned FP32 values (6e-8) lie below it.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

REL = 1e-6


def _rel(a, b):
    return np.linalg.norm(a.astype(np.float64) - b) / np.linalg.norm(b)


def _problem(kind, seed=3):
    rng = np.random.default_rng(seed)
    n = {"tiny": 37, "edges": 9_001, "long": 60_013}.get(kind, 20_011)
    inter = [None, None, None]
    if kind == "tiny":
        refs = [rng.integers(1, 9, n), rng.integers(1, 4, n)]
        nlev = [8, 3]
    elif kind == "edges":
        # primary levels of 1, 2, 123..126 and 250 rows, then empty ones
        sizes = [1, 2, 123, 124, 125, 126, 250] * 12
        r = np.repeat(np.arange(1, len(sizes) + 1), sizes)[:n]
        refs = [rng.permutation(r), rng.integers(1, 41, r.size)]
        n, nlev = r.size, [len(sizes) + 70, 45]
    elif kind == "long":
        # one primary level with a fifth of the rows, a few-level effect of pieces
        r = rng.integers(1, 3001, n)
        r[rng.random(n) < 0.2] = 7
        refs = [r, rng.integers(1, 601, n), rng.integers(1, 6, n)]
        nlev = [3000, 600, 5]
    elif kind == "four":
        refs = [rng.integers(1, 1501, n), rng.integers(1, 301, n), rng.integers(1, 51, n),
                rng.integers(1, 8, n)]
        nlev = [1500, 300, 50, 7]
        inter = [None, None, None, None]
    elif kind == "interacted":
        refs = [rng.integers(1, 2001, n), rng.integers(1, 201, n), rng.integers(1, 31, n)]
        nlev = [2000, 200, 30]
        inter = [None, None, rng.uniform(0.5, 1.5, n)]
    else:  # the primary effect interacted
        refs = [rng.integers(1, 201, n), rng.integers(1, 2001, n)]
        nlev = [200, 2000]
        inter = [None, rng.uniform(0.5, 1.5, n)]
    return n, [r.astype(np.int64) for r in refs], nlev, inter[:len(refs)], rng


def _solver(fe, refs, nlev, inter, w):
    return fe.AbstractFixedEffectSolver(
        [fe.FixedEffect.from_refs(r, m, a) for r, m, a in zip(refs, nlev, inter)], w, "CUDA",
        np.float32)


@pytest.mark.parametrize("kind", ["tiny", "edges", "long", "four", "interacted", "primary"])
@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("cols", [1, 2, 3, 8])
def test_matches_oracle(fe, oracle, kind, weighted, cols):
    n, refs, nlev, inter, rng = _problem(kind)
    w = rng.uniform(0.5, 1.5, n) if weighted else None
    Y = np.asfortranarray((rng.standard_normal((n, cols)) + (refs[0] % 7)[:, None] * 0.4)
                          .astype(np.float32))
    R_o, _, _ = oracle.solve_residuals_cols(Y.astype(np.float64), refs, nlev, inter, w, tol=1e-10)
    feM = _solver(fe, refs, nlev, inter, w)
    feM.set_option(fe._lib.FE_OPT_PROFILE, 1)
    R, its, cv = feM.solve_residuals(Y.copy(order="F"), tol=1e-8)
    assert "coef_solve" in feM.kernel_stats()
    feM.set_option(fe._lib.FE_OPT_PROFILE, 0)
    R2, its2, _ = feM.solve_residuals(Y.copy(order="F"), tol=1e-8)
    feM.close()
    assert cv.all() and R.dtype == np.float32
    assert np.array_equal(R, R2) and np.array_equal(its, its2)
    assert max(_rel(R[:, j], R_o[:, j]) for j in range(cols)) < REL


def test_weights_replaced_and_removed(fe, oracle):
    n, refs, nlev, inter, rng = _problem("interacted")
    y = (rng.standard_normal(n) + refs[1] % 5).astype(np.float32)
    feM = _solver(fe, refs, nlev, inter, None)
    for w in (None, rng.uniform(0.5, 1.5, n), rng.uniform(0.1, 9.0, n), None):
        feM.update_weights(w)
        r, _, cv = feM.solve_residuals(y.copy(), tol=1e-8)
        r_o = oracle.solve_residuals(y.astype(np.float64), refs, nlev, inter, w, tol=1e-10)[0]
        assert cv and _rel(r, r_o) < REL
    feM.close()


def test_zero_and_nan_columns(fe):
    # a zero column stops at once with a zero residual, a NaN column stops at
    # once unconverged; the others are solved as without them
    n, refs, nlev, inter, rng = _problem("long")
    Y = np.asfortranarray(rng.standard_normal((n, 5)).astype(np.float32))
    feM = _solver(fe, refs, nlev, inter, None)
    R0, its0, _ = feM.solve_residuals(Y.copy(order="F"), tol=1e-8)
    Y[:, 1] = 0.0
    Y[11, 3] = np.nan
    R, its, cv = feM.solve_residuals(Y.copy(order="F"), tol=1e-8)
    feM.close()
    assert list(cv) == [True, True, True, False, True]
    assert np.array_equal(R[:, 1], np.zeros(n)) and np.isnan(R[11, 3]) and its[3] <= 2
    for j in (0, 2, 4):
        assert np.array_equal(R[:, j], R0[:, j]) and its[j] == its0[j]


def test_exact_fit_takes_the_row_side(fe, oracle):
    # a column in the span of the effects (to FP32 rounding): the squared
    # residual norm cancels on the coefficient side, so the rows are formed
    n, refs, nlev, inter, rng = _problem("four")
    y = sum(rng.standard_normal(m + 1)[r] for r, m in zip(refs, nlev)).astype(np.float32)
    feM = _solver(fe, refs, nlev, inter, None)
    feM.set_option(fe._lib.FE_OPT_PROFILE, 1)
    r, _, cv = feM.solve_residuals(y.copy(), tol=1e-8)
    assert "demean64" in feM.kernel_stats()
    feM.close()
    r_o = oracle.solve_residuals(y.astype(np.float64), refs, nlev, inter, None, tol=1e-8)[0]
    assert cv and np.linalg.norm(r - r_o) < REL * np.linalg.norm(y)


def test_zero_weights_and_maxiter(fe):
    # an observation of weight 0 has no residual (0 / 0, as on the row side);
    # too few iterations are reported as not converged
    n, refs, nlev, inter, rng = _problem("long")
    w = rng.uniform(0.5, 1.5, n)
    w[::17] = 0.0
    y = rng.standard_normal(n).astype(np.float32)
    out = []
    for absorb in (1, 0):
        feM = _solver(fe, refs, nlev, inter, w)
        feM.set_option(fe._lib.FE_OPT_ABSORB, absorb)
        r, _, cv = feM.solve_residuals(y.copy(), tol=1e-8)
        assert cv and np.isnan(r[::17]).all()
        out.append(r[w > 0])
        r, it, cv = feM.solve_residuals(y.copy(), tol=1e-8, maxiter=3)
        assert not cv and it == 3
        feM.close()
    assert _rel(out[0], out[1].astype(np.float64)) < REL


@pytest.mark.parametrize("kind", ["tiny", "edges", "long", "four", "interacted", "primary"])
@pytest.mark.parametrize("weighted,cols", [(False, 1), (True, 1), (True, 3), (False, 8)])
def test_plain_loop_in_one_kernel(fe, oracle, kind, weighted, cols):
    # FP64 solves of narrow tiles: the loop in one cooperative kernel against
    # the launched loop (the same recurrences over sums in another order, so
    # equal counts and rounding-level differences, scaled by the few iterations
    # of these well-conditioned problems) and the oracle
    n, refs, nlev, inter, rng = _problem(kind)
    w = rng.uniform(0.5, 1.5, n) if weighted else None
    Y = np.asfortranarray(rng.standard_normal((n, cols)) + (refs[0] % 7)[:, None] * 0.4)
    fes = [fe.FixedEffect.from_refs(r, m, a) for r, m, a in zip(refs, nlev, inter)]
    out = []
    for launched in (False, True):
        feM = fe.AbstractFixedEffectSolver(fes, w, "CUDA", np.float64)
        if launched:
            feM.set_option(fe._lib.FE_OPT_EXPAND_VARIANT, 0)
            feM.set_option(fe._lib.FE_OPT_SEGSUM_VARIANT, 0)
        feM.set_option(fe._lib.FE_OPT_PROFILE, 1)
        R, its, cv = feM.solve_residuals(Y.copy(order="F"), tol=1e-8)
        assert ("plain_loop" in feM.kernel_stats()) != launched
        feM.set_option(fe._lib.FE_OPT_PROFILE, 0)
        R2, its2, _ = feM.solve_residuals(Y.copy(order="F"), tol=1e-8)
        b, it_b, cv_b = feM.solve_coefficients(Y[:, 0], tol=1e-8)
        feM.close()
        assert cv.all() and cv_b and np.array_equal(R, R2) and np.array_equal(its, its2)
        out.append((R, its, b, it_b))
    (R, its, b, it_b), (R1, its1, b1, it_b1) = out
    assert np.abs(its - its1).max() <= 1 and abs(it_b - it_b1) <= 1
    for j in range(cols):
        if its[j] == its1[j]:
            assert _rel(R[:, j], R1[:, j]) < 1e-10
    r_o, it_o, _ = oracle.solve_residuals(Y[:, 0], refs, nlev, inter, w, tol=1e-8)
    assert abs(int(its[0]) - int(it_o)) <= 1 and _rel(R[:, 0], r_o) < REL
    fit = [sum(x * (1.0 if a is None else a) for x, a in zip(c, inter)) for c in (b, b1)]
    assert np.linalg.norm(fit[0] - fit[1]) < REL * np.linalg.norm(fit[1])
