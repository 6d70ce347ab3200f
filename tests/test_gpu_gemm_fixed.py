"""The FP64-grade tensor-core kernel (gemm_multi.cu) at the edges of its tiles
(128 rows, 32 or 64 columns), of its stages of 32 K elements, of its chunks of
five stages and of its K splits: exact where the product is exact in FP64."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bn", [32, 64])
@pytest.mark.parametrize("M,N,K,ksplit", [(1, 1, 1, 1), (128, 64, 16, 1), (129, 65, 17, 1), (300, 33, 160, 1),
                                          (257, 31, 161, 1), (64, 200, 1000, 3), (1000, 70, 352, 1)])
def test_fixed_gemm_is_exact_where_the_product_is(gbcc_lib, M, N, K, ksplit, bn):
    # 18- and 16-bit integers under power-of-two row scales: sums of K <= 1000
    # products fit 44 bits
    rng = np.random.default_rng(M + N + K + bn)
    A = rng.integers(-(1 << 17), 1 << 17, size=(M, K)).astype(np.float64)
    B = rng.integers(-(1 << 15), 1 << 15, size=(N, K)).astype(np.float64)
    A *= np.ldexp(1.0, rng.integers(-20, 20, size=(M, 1)))
    B *= np.ldexp(1.0, rng.integers(-20, 20, size=(N, 1)))
    out = np.zeros((M, N))
    ms = C.c_float()
    st = gbcc_lib.gbcc_testing_gemm_fp64tc(M, N, K, A.ctypes.data, B.ctypes.data, out.ctypes.data, bn, ksplit, 0, 1,
                                           C.byref(ms))
    assert st == 0
    assert np.array_equal(out, A @ B.T)
