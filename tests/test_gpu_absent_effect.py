"""One-problem plans with an effect that has no levels (level ids 0): solved as
without that effect, on every route that a narrow tile can take.

The bar is the repository's 1e-6 on the residual's relative 2-norm (FP32
columns round at 6e-8, the solves stop at 1e-8).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

REL = 1e-6
N = 5_003
LEVELS = (400, 60, 9)


def _refs(seed=4):
    rng = np.random.default_rng(seed)
    return [rng.integers(1, m + 1, N) for m in LEVELS], rng


def _effects(fe, refs, absent):
    """The effects, with one of no levels inserted at position `absent`."""
    fes = [fe.FixedEffect.from_refs(r, m) for r, m in zip(refs, LEVELS)]
    fes.insert(absent, fe.FixedEffect.from_refs(np.zeros(N, dtype=np.int64), 0))
    return fes


@pytest.mark.parametrize("T", [np.float32, np.float64])
@pytest.mark.parametrize("present,absent", [(1, 1), (2, 0), (2, 1), (2, 2), (3, 1)])
@pytest.mark.parametrize("weighted", [False, True])
def test_residuals_as_without_the_absent_effect(fe, oracle, T, present, absent, weighted):
    refs, rng = _refs()
    refs, nlev = refs[:present], list(LEVELS[:present])
    w = rng.uniform(0.5, 1.5, N) if weighted else None
    Y = np.asfortranarray((rng.standard_normal((N, 3)) + (refs[0] % 5)[:, None]).astype(T))
    R_o, _, _ = oracle.solve_residuals_cols(Y.astype(np.float64), refs, nlev, [None] * present, w,
                                            tol=1e-10)
    fes = _effects(fe, refs, absent)
    feM = fe.AbstractFixedEffectSolver(fes, w, "CUDA", T)
    R, _, cv = feM.solve_residuals(Y.copy(order="F"), tol=1e-8)
    feM.close()
    bs = fe.BatchSolver([fes], None if w is None else [w], T)
    r, _, cvb = bs.solve_residuals([Y[:, 0].copy()], tol=1e-8)
    bs.close()
    assert cv.all() and cvb.all()
    for a, b in [(R[:, j], R_o[:, j]) for j in range(3)] + [(r[0], R_o[:, 0])]:
        assert np.linalg.norm(a.astype(np.float64) - b) < REL * np.linalg.norm(b)


def test_coefficients_as_without_the_absent_effect(fe):
    # the fitted values, which unlike the coefficients are unique
    refs, rng = _refs()
    y = rng.standard_normal(N) + refs[0] % 5
    fit = []
    for absent in (None, 1):
        fes = _effects(fe, refs[:2], 1)
        if absent is None:
            del fes[1]
        L = fe._lib.load()
        feM = fe.AbstractFixedEffectSolver(fes, None, "CUDA", np.float64)
        coefs = [np.zeros(max(f.n, 1)) for f in fes]
        it, cv = np.zeros(1, dtype=np.int64), np.zeros(1, dtype=np.uint8)
        fe._lib.check(L.fe_solve_coefficients(
            feM._h, y.ctypes.data, fe._lib.FE_DTYPE_F64, fe._lib.FE_PREC_FP64, 1e-8, 10_000,
            fe._ptrs(coefs), it.ctypes.data_as(fe._lib._i64p), cv.ctypes.data_as(fe._lib._u8p)))
        feM.close()
        assert cv[0]
        fit.append(sum(c[f.refs - 1] for c, f in zip(coefs, fes) if f.n))
    assert np.linalg.norm(fit[0] - fit[1]) < REL * np.linalg.norm(fit[0])
