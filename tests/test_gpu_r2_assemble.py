"""The last pass of r2 against its definition: edges of the per-pair kernel (one
occupied or virtual orbital, odd and even rows, several elements a thread) and
of its largest o (64, 68), and the tiled kernel past it (69)."""
import ctypes

import numpy as np
import pytest

from mpqc_gb300 import _lib

pytestmark = pytest.mark.gpu


def unpack(Bp, Bm, o, v):
    out = np.empty((v, v, o, o))
    su, au = np.triu_indices(o), np.triu_indices(o, 1)
    p = m = 0
    for a in range(v):
        for b in range(a, v):
            X = np.zeros((o, o))
            X[su] = Bp[p]
            X.T[su] = Bp[p]
            p += 1
            if b > a:
                if Bm is not None:
                    X[au] += Bm[m]
                    X.T[au] -= Bm[m]
                m += 1
            out[a, b], out[b, a] = X, X.T
    return out


@pytest.mark.parametrize("pairs,acc", [(2, 0), (1, 0), (0, 1)])
@pytest.mark.parametrize("o,v", [(1, 1), (1, 3), (2, 1), (5, 4), (13, 9), (33, 3), (64, 2), (68, 2), (69, 2)])
def test_assembly_is_its_definition(o, v, pairs, acc):
    lib = _lib.load()
    rng = np.random.default_rng(o + 100 * v + pairs)
    u, t, g, r = (rng.normal(size=(v, v, o, o)) for _ in range(4))
    Bp = rng.normal(size=(v * (v + 1) // 2, o * (o + 1) // 2)) if pairs else None
    Bm = rng.normal(size=(v * (v - 1) // 2, o * (o - 1) // 2)) if pairs == 2 and o > 1 and v > 1 else None
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
