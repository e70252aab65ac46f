"""Allocations that fail (injected on the host) where another way is left."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N, LEVELS = 200_003, (20_000, 300, 50)


def _effects(fe):
    rng = np.random.default_rng(5)
    fes = [fe.FixedEffect.from_refs(rng.integers(1, m + 1, N), m) for m in LEVELS]
    return fes, rng.standard_normal(N)


@pytest.mark.parametrize("T", [np.float32, np.float64])
def test_a_failed_pool_request_becomes_a_block_of_its_own(fe, monkeypatch, T):
    fes, y = _effects(fe)
    ref, _, _ = fe.AbstractFixedEffectSolver(fes, None, "CUDA", T).solve_residuals(y.astype(T))
    monkeypatch.setenv("FE_B200_FAIL_POOL_BYTES", "1000")
    feM = fe.AbstractFixedEffectSolver(fes, None, "CUDA", T)
    r, _, cv = feM.solve_residuals(y.astype(T))
    feM.close()
    assert cv and np.array_equal(r, ref)


def test_a_failed_allocation_takes_what_the_pool_keeps(fe, monkeypatch):
    import torch
    fes, y = _effects(fe)
    fe.AbstractFixedEffectSolver(fes, None, "CUDA", np.float32).close()
    torch.cuda.synchronize()
    kept = torch.cuda.mem_get_info()[0]
    monkeypatch.setenv("FE_B200_FAIL_ALLOC_BYTES", "1")  # no block of the pool is in use
    with pytest.raises(RuntimeError):
        fe.AbstractFixedEffectSolver(fes, None, "CUDA", np.float32)
    # the plan's refs alone were 8 x 200 kB
    assert torch.cuda.mem_get_info()[0] > kept + (1 << 20)


def _loops(fe, feM, launched):
    feM.set_option(fe._lib.FE_OPT_EXPAND_VARIANT, 0 if launched else -1)


@pytest.mark.parametrize("T,kernel", [(np.float32, "coef_solve"), (np.float64, "plain_loop")])
def test_without_room_for_its_arrays_a_solve_takes_the_launched_loops(fe, monkeypatch, T, kernel):
    fes, y = _effects(fe)
    feM = fe.AbstractFixedEffectSolver(fes, None, "CUDA", T)
    feM.set_option(fe._lib.FE_OPT_PROFILE, 1)
    _loops(fe, feM, True)  # the launched loops' workspace is there
    ref, _, _ = feM.solve_residuals(y.astype(T), tol=1e-8)
    _loops(fe, feM, False)
    monkeypatch.setenv("FE_B200_FAIL_ALLOC_BYTES", "100000")
    r, _, cv = feM.solve_residuals(y.astype(T), tol=1e-8)
    assert cv and kernel not in feM.kernel_stats()
    assert np.linalg.norm(r - ref) < 1e-6 * np.linalg.norm(ref)
    monkeypatch.delenv("FE_B200_FAIL_ALLOC_BYTES")
    r, _, cv = feM.solve_residuals(y.astype(T), tol=1e-8)
    assert cv and kernel in feM.kernel_stats()
    feM.close()


@pytest.mark.parametrize("T,cols", [(np.float32, 3), (np.float64, 3)])
def test_the_launched_loops_take_the_room_of_the_coefficient_side(fe, monkeypatch, T, cols):
    # the first large allocation of the launched loops fails while the other
    # side's arrays are held, and the one of the host columns' copy as well
    fes, y = _effects(fe)
    Y = np.asfortranarray(np.repeat(y[:, None], cols, axis=1).astype(T))
    feM = fe.AbstractFixedEffectSolver(fes, None, "CUDA", T)
    ref, _, _ = feM.solve_residuals(Y.copy(order="F"), tol=1e-8)
    _loops(fe, feM, True)
    monkeypatch.setenv("FE_B200_FAIL_ALLOC_BYTES", "100000/1")
    Y2 = np.asfortranarray(np.concatenate([Y] * 6, axis=1))
    r, _, cv = feM.solve_residuals(Y2, tol=1e-8)
    assert cv.all() and np.linalg.norm(r[:, 0] - ref[:, 0]) < 1e-6 * np.linalg.norm(ref[:, 0])
    feM.close()
    feM = fe.AbstractFixedEffectSolver(fes, None, "CUDA", T)
    feM.solve_residuals(Y.copy(order="F"), tol=1e-8)
    _loops(fe, feM, True)
    monkeypatch.setenv("FE_B200_FAIL_ALLOC_BYTES", "100000/01")
    r, _, cv = feM.solve_residuals(Y[:, :1].copy(order="F"), tol=1e-8)
    assert cv.all() and np.linalg.norm(r[:, 0] - ref[:, 0]) < 1e-6 * np.linalg.norm(ref[:, 0])
    feM.close()
