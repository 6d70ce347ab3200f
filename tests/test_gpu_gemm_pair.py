"""The split-BF16 GEMM on CTA pairs (gemm_pair.cu: 256 x 256 tiles, every slice
of a K block per stage) against FP64: edges of its tiles, short and ragged K,
K splits, band order, accumulating and column-major outputs."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# error of the split (2^-17, 2^-24 per element) plus FP32 chunk sums
SPLIT = {2: 3e-5, 3: 2e-6}


def _run(lib, A, B, slices, ksplit=1, group=1, cmode=0, chunk=0):
    M, K = A.shape
    N = B.shape[0]
    out = np.empty((M, N))
    ms = C.c_float()
    st = lib.gbcc_testing_gemm_ex3(M, N, K, A.ctypes.data, B.ctypes.data, out.ctypes.data, slices, ksplit, 256, 0,
                                   chunk, 0, 2, group, cmode, 1, C.byref(ms))
    assert st == 0
    return out


@pytest.mark.parametrize("slices,chunk", [(2, 24), (2, 4), (3, 4)])
@pytest.mark.parametrize("M,N,K,ksplit", [(1, 1, 1, 1), (128, 256, 64, 1), (129, 257, 33, 1), (700, 900, 384, 3),
                                          (513, 511, 1000, 1), (2000, 300, 100, 1)])
def test_pair_gemm_matches_fp64(gbcc_lib, M, N, K, ksplit, slices, chunk):
    rng = np.random.default_rng(M + N + K)
    A, B = rng.normal(size=(M, K)), rng.normal(size=(N, K))
    ref = A @ B.T
    out = _run(gbcc_lib, A, B, slices, ksplit, chunk=chunk)
    tol = SPLIT[slices] + 8 * 2.0 ** -24 * np.sqrt(K)
    assert np.max(np.abs(out - ref)) <= tol * max(np.max(np.abs(ref)), 1e-3)


@pytest.mark.parametrize("slices", [2, 3])
@pytest.mark.parametrize("ksplit", [1, 2])
def test_pair_gemm_forms_agree(gbcc_lib, slices, ksplit):
    """Band order, accumulation into zeros and a column-major C change no bits."""
    rng = np.random.default_rng(slices + ksplit)
    A, B = rng.normal(size=(1500, 512)), rng.normal(size=(1900, 512))
    ref = _run(gbcc_lib, A, B, slices, ksplit)
    for group, cmode in ((4, 0), (1, 1), (1, 2), (3, 3)):
        assert np.array_equal(ref, _run(gbcc_lib, A, B, slices, ksplit, group, cmode))
