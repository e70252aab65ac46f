"""The buffers that a sharded plan hands to its exchange callback are device
allocations of their own, whatever their size: other processes can open them
(cudaIpcGetMemHandle), which memory of a pool does not allow."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

IS_LEGACY_CUDA_IPC_CAPABLE = 10  # CUpointer_attribute


@pytest.mark.parametrize("prec,cols", [("fp64", 1), ("mixed", 1), ("mixed", 32)])
def test_exchange_buffers_can_be_shared(fe, prec, cols):
    cuda = ctypes.CDLL("libcuda.so.1")
    seen = []

    def exchange(ctx, buf, count, dtype, stream):  # one rank: the sum is what is there
        v = ctypes.c_int(-1)
        rc = cuda.cuPointerGetAttribute(ctypes.byref(v), IS_LEGACY_CUDA_IPC_CAPABLE,
                                        ctypes.c_uint64(buf))
        seen.append((count, rc, v.value))
        return 0

    cb = fe._lib.EXCHANGE_FN(exchange)
    rng = np.random.default_rng(3)
    n, nlev = 30_011, np.array([3000, 300, 11], dtype=np.int64)
    refs = [rng.integers(1, m + 1, n) for m in nlev]
    L, h = fe._lib.load(), ctypes.c_void_p()
    fe._lib.check(L.fe_plan_create_sharded(ctypes.byref(h), n, 3, fe._ptrs(refs),
                                           nlev.ctypes.data_as(fe._lib._i64p), None, None, 0, cb,
                                           None))
    Y = np.asfortranarray(rng.standard_normal((n, cols)))
    its, cv = np.zeros(cols, dtype=np.int64), np.zeros(cols, dtype=np.uint8)
    fe._lib.check(L.fe_solve_residuals(
        h, Y.ctypes.data, fe._lib.FE_DTYPE_F64, cols, n,
        fe._lib.FE_PREC_FP64 if prec == "fp64" else fe._lib.FE_PREC_MIXED, 1e-8, 1000,
        its.ctypes.data_as(fe._lib._i64p), cv.ctypes.data_as(fe._lib._u8p)))
    fe._lib.check(L.fe_plan_destroy(h))
    assert cv.all() and seen
    assert all(rc == 0 and v == 1 for _, rc, v in seen), seen[:4]
