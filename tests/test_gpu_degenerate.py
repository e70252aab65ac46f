"""Effects that add nothing to another one (a single level, levels nested in the
first effect's), alone and beside others, with right-hand sides that the
coefficient side has to hand over: against the residual by dense projection.

The bar is the repository's 1e-6, of the residual or, for columns that the
effects fit or that have a large mean, of the column in FP32 (3 roundings of
6e-8 and the solve's own).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

REL = 1e-6


def _dense(refs, nlev, w, Y):
    n = Y.shape[0]
    X = np.concatenate([np.eye(m)[r - 1] for r, m in zip(refs, nlev)], axis=1)
    sw = np.ones(n) if w is None else np.sqrt(w)
    U, s, _ = np.linalg.svd(sw[:, None] * X, full_matrices=False)
    U = U[:, s > 1e-10 * s[0]]
    R = sw[:, None] * Y
    for _ in range(2):
        R = R - U @ (U.T @ R)
    return R / sw[:, None]


@pytest.mark.parametrize("kind", ["single", "singles", "nested", "nested_and_other", "tiny"])
@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("what", ["plain", "mean", "exact", "zero", "small"])
@pytest.mark.parametrize("cols", [1, 5])
def test_redundant_effects(fe, kind, weighted, what, cols):
    rng = np.random.default_rng(17)
    n = 5 if kind == "tiny" else 301
    first = rng.integers(1, (2 if kind == "tiny" else 30) + 1, n)
    ones = np.ones(n, dtype=np.int64)
    refs, nlev = {"single": ([first, ones], [30, 1]),
                  "singles": ([ones, ones, ones], [1, 1, 1]),
                  "nested": ([first, (first - 1) % 7 + 1], [30, 7]),
                  "nested_and_other": ([first, (first - 1) % 7 + 1, rng.integers(1, 6, n)],
                                       [30, 7, 5]),
                  "tiny": ([first, ones], [2, 1])}[kind]
    w = rng.uniform(0.5, 1.5, n) if weighted else None
    Y = rng.standard_normal((n, cols))
    if what == "mean":
        Y[:, 0] += 1e5
    elif what == "exact":
        Y[:, 0] = sum(rng.standard_normal(m + 1)[r] for r, m in zip(refs, nlev))
    elif what == "zero":
        Y[:, 0] = 0
    elif what == "small":
        Y[:, 0] *= 1e-18
    Y = np.asfortranarray(Y.astype(np.float32))
    feM = fe.AbstractFixedEffectSolver(
        [fe.FixedEffect.from_refs(r, m) for r, m in zip(refs, nlev)], w, "CUDA", np.float32)
    R, its, cv = feM.solve_residuals(Y.copy(order="F"), tol=1e-8, maxiter=2000)
    feM.close()
    T = _dense(refs, nlev, w, Y.astype(np.float64))
    for j in range(cols):
        loose = j == 0 and what in ("mean", "exact")
        bar = REL * np.linalg.norm(Y[:, 0] if loose else T[:, j])
        assert np.linalg.norm(R[:, j] - T[:, j]) <= bar, (j, its[j], cv[j])
        if not loose:
            assert cv[j], (j, its[j])
            # (beside an exact column the row side may solve the tile, whose
            # FP32 inner solves take hundreds of iterations on nested effects)
            assert its[j] < 60 or what == "exact", (j, its[j])
