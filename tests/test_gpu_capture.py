"""Plans built, solved and freed on one thread while another thread captures a
graph: the capture stays valid, and so do the plans' results.  (Waiting for the
whole device would end the capture.)"""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _problem(fe, n=30_011, cols=16, seed=2):
    rng = np.random.default_rng(seed)
    fes = [fe.FixedEffect.from_refs(rng.integers(1, m + 1, n), m) for m in (3000, 300, 11)]
    return fes, np.asfortranarray(rng.standard_normal((n, cols)).astype(np.float32))


def _solve(fe, fes, Y, T=np.float32):
    feM = fe.AbstractFixedEffectSolver(fes, None, "CUDA", T)
    try:
        R, _, cv = feM.solve_residuals(Y.astype(T, order="F"), tol=1e-8)
    finally:
        feM.close()
    assert cv.all()
    return R


def _thread(errors, f):
    def run():
        try:
            f()
        except BaseException as e:  # noqa: BLE001  (reported by the caller)
            errors.append(e)
    t = threading.Thread(target=run)
    t.start()
    return t


@pytest.mark.parametrize("T,cols", [(np.float32, 16), (np.float32, 2), (np.float64, 1)])
def test_a_callers_capture_survives_plans_of_another_thread(fe, T, cols):
    import torch
    fes, Y = _problem(fe, cols=cols)
    ref = _solve(fe, fes, Y, T)
    a = torch.arange(1000, dtype=torch.float32, device="cuda")
    out, errors = [], []
    g, s = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(s):
        g.capture_begin(capture_error_mode="thread_local")
        b = a * 2
        t = _thread(errors, lambda: out.append(_solve(fe, fes, Y, T)))
        t.join()
        c = b + 1
        g.capture_end()
    g.replay()
    torch.cuda.synchronize()
    assert not errors, errors
    assert np.array_equal(out[0], ref)
    assert torch.equal(c, a * 2 + 1)


def test_captured_loops_survive_plans_of_other_threads(fe):
    # 16 columns: the loop is captured by every new plan's first solve
    fes, Y = _problem(fe)
    ref = _solve(fe, fes, Y)
    small = _problem(fe, 4_001, 1, 3)
    stop, errors, bad = threading.Event(), [], []

    def churn():
        while not stop.is_set():
            _solve(fe, *small)

    def solves():
        for _ in range(25):
            if not np.array_equal(_solve(fe, fes, Y), ref):
                bad.append(1)

    others = [_thread(errors, churn) for _ in range(2)]
    mine = [_thread(errors, solves) for _ in range(2)]
    for t in mine:
        t.join()
    stop.set()
    for t in others:
        t.join()
    assert not errors, errors
    assert not bad


def test_scales_on_a_callers_stream_before_the_plan_ends(fe):
    # the scales are computed from the plan's arrays on the caller's stream,
    # which is still busy when the plan is freed and its memory reused
    import ctypes
    import torch
    fes, _ = _problem(fe)
    feM = fe.AbstractFixedEffectSolver(fes, np.linspace(0.5, 1.5, 30_011), "CUDA", np.float64)
    ref = feM.scales()
    L, s = fe._lib.load(), torch.cuda.Stream()
    out = torch.empty(3000, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    with torch.cuda.stream(s):
        torch.cuda._sleep(20_000_000)
    fe._lib.check(L.fe_plan_scales_noalloc(feM._h, 0, ctypes.c_void_p(out.data_ptr()),
                                           ctypes.c_void_p(s.cuda_stream)))
    feM.close()
    other = fe.AbstractFixedEffectSolver(fes, np.linspace(9.0, 2.0, 30_011), "CUDA", np.float64)
    torch.cuda.synchronize()
    other.close()
    assert np.allclose(out.cpu().numpy(), ref[0], rtol=1e-13, atol=0)


def test_a_device_solve_while_a_blocking_stream_is_captured(fe):
    # such a capture forbids the use of the default stream to everyone; the
    # solve runs on the plan's own stream
    import ctypes
    import torch
    rt = ctypes.CDLL("libcudart.so.12")
    fes, Y = _problem(fe, cols=1)
    feM = fe.AbstractFixedEffectSolver(fes, None, "CUDA", np.float32)
    y = torch.from_numpy(Y[:, 0].copy()).cuda()
    ref = feM.solve_residuals(y.clone(), tol=1e-8)[0].cpu()
    work = y.clone()
    h, graph = ctypes.c_void_p(), ctypes.c_void_p()
    buf = torch.zeros(1000, device="cuda")
    torch.cuda.synchronize()
    assert rt.cudaStreamCreate(ctypes.byref(h)) == 0
    assert rt.cudaStreamBeginCapture(h, 1) == 0  # cudaStreamCaptureModeThreadLocal
    assert rt.cudaMemsetAsync(ctypes.c_void_p(buf.data_ptr()), 0, 4000, h) == 0
    errors, out = [], []
    t = _thread(errors, lambda: out.append(feM.solve_residuals(work, tol=1e-8)))
    t.join()
    rc = rt.cudaStreamEndCapture(h, ctypes.byref(graph))
    if rc == 0:
        rt.cudaGraphDestroy(graph)
    rt.cudaGetLastError()
    rt.cudaStreamDestroy(h)
    feM.close()
    assert rc == 0 and not errors, (rc, errors)
    assert torch.equal(out[0][0].cpu(), ref)
