"""GEMM with the reduction in slices: a last slice shorter than the others, ragged in 32 and in 4, results off the vector width, bias added once,
either operand transposed, against numpy FP64."""
import ctypes

import numpy as np
import pytest

import b200conv
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [(128, 64, 64), (128, 64, 128), (320, 320, 8000), (2048, 512, 4096), (130, 70, 1025), (512, 768, 3072), (128, 1000, 999),
                                   (1, 1, 128), (16, 64, 128), (63, 65, 127), (100, 1000, 2048), (300, 33, 1031), (17, 4096, 143),
                                   (2500, 2304, 64), (20500, 128, 96)])
@pytest.mark.parametrize("ta,tb", [(False, False), (True, False), (False, True)])
def test_sliced_reduction(m, n, k, ta, tb):
    rng = np.random.default_rng(m + n + k)
    a, b, bias = rng.standard_normal((m, k), dtype=np.float32), rng.standard_normal((k, n), dtype=np.float32), rng.standard_normal(n, dtype=np.float32)
    va, vb, vbias = b200conv.DeviceView(np.ascontiguousarray(a.T) if ta else a), b200conv.DeviceView(np.ascontiguousarray(b.T) if tb else b), b200conv.DeviceView(bias)
    out = b200conv.DeviceBuffer(4 * m * n)
    f = ctypes.c_float
    b200conv.check(b200conv.lib().b200_gemm(m, n, k, va.ptr, *((1, m) if ta else (k, 1)), vb.ptr, *((1, k) if tb else (n, 1)), vbias.ptr, f(0.5), f(2.0),
                                            out.ptr, b200conv.ALGO_AUTO, None))
    assert b200conv.last_kernel() == ("tc_gemm" if m >= 128 and n >= 64 else "simt_gemm") and b200conv.device_status() == 0
    want = 0.5 * (a.astype(np.float64) @ b.astype(np.float64)) + 2.0 * bias
    assert oracle.rel_l2(out.to_numpy((m, n)), want) <= 1e-5
