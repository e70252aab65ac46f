"""Order of device-buffer solves against the caller's streams."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_device_columns_wait_for_the_default_stream(fe):
    # device columns written on the default stream just before the call: the
    # solve on the plan's own (non-blocking) stream reads them, not what the
    # buffer held before
    import torch
    rng = np.random.default_rng(3)
    n = 20_011
    fes = [fe.FixedEffect(rng.integers(1, m + 1, n)) for m in (2000, 200)]
    y = torch.from_numpy(rng.standard_normal(n).astype(np.float32)).cuda()
    feM = fe.AbstractFixedEffectSolver(fes, None, "CUDA", np.float32)
    ref, _, _ = feM.solve_residuals(y.clone(), tol=1e-8)
    torch.cuda.synchronize()
    work = torch.zeros_like(y)
    torch.cuda.synchronize()
    torch.cuda._sleep(40_000_000)  # about 20 ms of the default stream
    work.copy_(y)
    r, _, _ = feM.solve_residuals(work, tol=1e-8)
    feM.close()
    assert torch.equal(r, ref)
