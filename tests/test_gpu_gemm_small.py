"""The in-place FP64 kernel of small contractions (gemm_small.cu) against the
FP64 product: edges of its output tiles (16 wide, 64 or 256 / 16 rows), K
lanes, staged steps of 32, and the split of K over blocks."""
import ctypes

import numpy as np
import pytest

from mpqc_gb300 import _lib

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 1), (5, 5, 9025), (16, 16, 32), (17, 16, 33), (57, 13, 13), (64, 1, 31), (65, 1, 741),
          (95, 95, 95), (190, 15, 190), (257, 17, 64), (1000, 31, 7), (13, 13, 42237)]


@pytest.mark.parametrize("mode", range(16))
@pytest.mark.parametrize("M,N,K", SHAPES)
def test_small_gemm_is_the_fp64_product(M, N, K, mode):
    lib = _lib.load()
    rng = np.random.default_rng(M + 7 * N + 13 * K)
    A, B, C = rng.normal(size=(M, K)), rng.normal(size=(N, K)), rng.normal(size=(M, N))
    Ain = np.ascontiguousarray(A.T) if mode & 1 else A
    Bin = np.ascontiguousarray(B.T) if mode & 2 else B
    scale = (-0.5 if mode & 4 else 1.0) * (1.25 if mode & 8 else 1.0)
    ref = scale * (A @ B.T) + (C if mode & 4 else 0.0)
    out = C.copy()
    ms = ctypes.c_float()
    st = lib.gbcc_testing_gemm_small(M, N, K, Ain.ctypes.data, Bin.ctypes.data, out.ctypes.data, mode, 1,
                                     ctypes.byref(ms))
    assert st == 0
    # a sum of K products in any order: K ulps of the sum of their magnitudes
    bound = 2.0 ** -52 * (K + 4) * (np.abs(scale) * (np.abs(A) @ np.abs(B).T) + np.abs(C))
    assert np.all(np.abs(out - ref) <= bound)
