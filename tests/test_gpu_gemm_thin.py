"""Tensor-core tiles whose sum stays in FP32 (few chunks of K): the split product
against FP64 at the edges of the tiles and of the epilogue's 16-column groups,
and the same bits in every output form and K split into one."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(lib, A, B, bn, sps, cmode):
    M, K = A.shape
    N = B.shape[0]
    out = np.empty((M, N))
    st = lib.gbcc_testing_gemm_ex3(M, N, K, A.ctypes.data, B.ctypes.data, out.ctypes.data, 2, 1, bn, 0, 0, 0, sps, 1,
                                   cmode, 1, C.byref(C.c_float()))
    assert st == 0
    return out


@pytest.mark.parametrize("bn,sps", [(32, 1), (64, 1), (64, 2), (128, 2), (192, 1), (256, 1)])
@pytest.mark.parametrize("M,N,K", [(1, 1, 1), (127, 15, 50), (129, 17, 190), (300, 63, 64), (128, 64, 65),
                                   (257, 65, 128), (20000, 50, 190), (640, 193, 30)])
def test_short_products(gbcc_lib, M, N, K, bn, sps):
    rng = np.random.default_rng(M + N + K)
    A, B = rng.normal(size=(M, K)), rng.normal(size=(N, K))
    ref = A @ B.T
    out = _run(gbcc_lib, A, B, bn, sps, 0)
    # two BF16 slices: 2^-17 an element and the dropped pair, and FP32 chunk sums
    tol = 3e-5 + 8 * 2.0 ** -24 * np.sqrt(K)
    assert np.max(np.abs(out - ref)) <= tol * max(np.max(np.abs(ref)), 1e-3)
    for cmode in (1, 2, 3):
        assert np.array_equal(out, _run(gbcc_lib, A, B, bn, sps, cmode))
