"""The rule that sends an FP64 product to the tensor cores or to the FMA kernel, against measured times of
both (one GB300, us, a call's overhead included): wherever one of them takes more than 1.1 times as long as
the other, the rule takes the faster one.  The rule needs nothing but the number of SMs.
"""
import ctypes

import numpy as np
import pytest

# m, n, k, FMA, tensor cores
MEASURED = [(48, 48, 15360, 92.4, 112.7), (24, 24, 2880, 32.5, 60.6), (30, 30, 9000, 45.4, 85.0),
            (36, 36, 6480, 55.1, 80.4), (48, 48, 8000, 58.5, 82.6), (72, 72, 25000, 325.2, 170.2),
            (72, 72, 45000, 560.7, 269.6), (96, 96, 60000, 979.4, 355.4), (120, 120, 180000, 4965.3, 1221.0),
            (64, 64, 4096, 58.3, 60.4), (64, 64, 32768, 288.4, 194.9), (64, 64, 100000, 822.5, 514.7),
            (128, 64, 16384, 253.9, 120.4), (128, 128, 16384, 480.5, 126.9), (128, 128, 65536, 1828.8, 403.1),
            (200, 200, 20000, 1447.5, 181.6), (256, 128, 30000, 1630.8, 231.7), (20, 20, 200000, 460.0, 951.1),
            (16, 16, 500000, 1102.3, 2707.7), (300, 64, 9000, 318.3, 105.7), (480, 480, 480, 219.7, 58.2),
            (216, 216, 600, 79.1, 53.9), (128, 128, 3600, 128.8, 61.4), (128, 400, 3600, 335.4, 71.1),
            (400, 128, 3600, 336.6, 72.9)]


@pytest.fixture(scope="module")
def pays():
    from quack_gb300 import build
    f = getattr(ctypes.CDLL(build.build()), "_Z15qk_gemm_tc_paysPK6qk_ctxiiii")
    f.restype = ctypes.c_bool
    ctx = np.zeros(4096, dtype=np.int32)      # a context's first members are the device and its SMs
    ctx[1] = 152
    return lambda m, n, k: f(ctx.ctypes.data_as(ctypes.c_void_p), m, n, k, 1)


@pytest.mark.parametrize("m,n,k,fma,tc", MEASURED)
def test_rule_takes_the_faster_kernel(pays, m, n, k, fma, tc):
    if max(fma, tc) > 1.1 * min(fma, tc):
        assert pays(m, n, k) == (tc < fma)
