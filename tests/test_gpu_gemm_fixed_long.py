"""FP64-grade tensor-core products over long K (gemm_multi.cu): sums of one sign,
whose float-float words grow with K, are exact where the product is exact in
FP64; at the edges of the windows of 32000 elements, and with K splits longer
than one."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bn", [32, 64])
@pytest.mark.parametrize("M,N,K,ksplit", [(300, 200, 2000, 1), (64, 300, 4096, 4), (5, 70, 16161, 1), (130, 66, 65536, 1), (1, 1, 32000, 1),
                                          (129, 65, 32001, 1), (33, 31, 262144, 1), (8, 40, 400000, 3)])
def test_long_sums_of_one_sign_are_exact(gbcc_lib, M, N, K, ksplit, bn):
    # 17- and 15-bit integers: sums of at most 400000 products stay below 2^51
    rng = np.random.default_rng(M + N + K)
    A = rng.integers(0, 1 << 17, size=(M, K)).astype(np.float64)
    B = rng.integers(0, 1 << 15, size=(N, K)).astype(np.float64)
    out = np.zeros((M, N))
    ms = C.c_float()
    st = gbcc_lib.gbcc_testing_gemm_fp64tc(M, N, K, A.ctypes.data, B.ctypes.data, out.ctypes.data, bn, ksplit, 0, 1,
                                           C.byref(ms))
    assert st == 0
    assert np.array_equal(out, A @ B.T)
