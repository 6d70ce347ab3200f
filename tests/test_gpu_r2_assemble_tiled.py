"""The last pass of r2 on both sides of the line between its kernels, wherever the
line lies: the per-pair kernel at its largest o, the tiled one just past it and at
o of other remainders to its tiles of 32."""
import ctypes

import numpy as np
import pytest

from mpqc_gb300 import _lib
from test_gpu_r2_assemble import unpack

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("v", [1, 2, 3])
@pytest.mark.parametrize("past", [0, 1, 2, 11, 28])
@pytest.mark.parametrize("pairs,acc", [(2, 0), (2, 1), (1, 0), (0, 1), (0, 0)])
def test_assembly_past_the_per_pair_kernel(v, past, pairs, acc):
    lib = _lib.load()
    o = lib.gbcc_testing_r2_assemble_pair_max(1 if pairs else 0) + past
    rng = np.random.default_rng(o + 100 * v + pairs)
    u, t, g, r = (rng.normal(size=(v, v, o, o)) for _ in range(4))
    Bp = rng.normal(size=(v * (v + 1) // 2, o * (o + 1) // 2)) if pairs else None
    Bm = rng.normal(size=(v * (v - 1) // 2, o * (o - 1) // 2)) if pairs == 2 and v > 1 else None
    q = u - 0.5 * t - t.transpose(1, 0, 2, 3)
    ref = q + q.transpose(1, 0, 3, 2) + g + (r if acc else 0.0)
    if pairs:
        ref = ref + unpack(Bp, Bm, o, v)
    out = r.copy()
    p = lambda x: ctypes.c_void_p(0 if x is None else x.ctypes.data)
    st = lib.gbcc_testing_r2_assemble(ctypes.c_int64(o), ctypes.c_int64(v), p(u), p(t), p(g), p(Bp), p(Bm), acc,
                                      p(out), 1, None)
    assert st == 0
    # eleven additions of values below 8 in any order
    assert np.abs(out - ref).max() <= 11 * 2.0 ** -52 * 32
