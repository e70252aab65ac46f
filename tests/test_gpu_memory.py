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
