"""Lanes of the residual program: the same bits in four lanes as in one, with and
without graphs; one lane where the device is short of memory; and workspaces that
are given up for (T) when it is short of memory come back."""
import ctypes as C

import numpy as np
import pytest

from conftest import ints_dict
from mpqc_gb300 import Solver, _lib, synth
from mpqc_gb300._lib import GBCC_ERR_OOM, GbccError

pytestmark = pytest.mark.gpu

FOUR = ("Fia", "Fij", "Fab", "Gijab", "Gijkl", "Giajb", "Gijka")


def make(method, o, v, **kw):
    """A handle of the method with its inputs, and amplitudes."""
    rng = np.random.default_rng(100 * o + v)
    n = o + v
    B = synth.make_df_factor(rng, 20, n, 0.05)
    if method == "direct":
        Cm = np.linalg.qr(rng.normal(size=(n, n)))[0]
        Bao, B = B, np.einsum("pi,Kpq,qj->Kij", Cm, B, Cm, optimize=True)
    eps_o, eps_v = np.sort(rng.uniform(-1.5, -0.3, size=o)), np.sort(rng.uniform(0.1, 3.0, size=v))
    t2 = rng.normal(0.0, 1e-2, size=(v, v, o, o))
    t2 = 0.5 * (t2 + t2.transpose(1, 0, 3, 2))
    inp = synth.inputs_from_factor(B, eps_o, eps_v, rng.normal(0.0, 1e-2, size=(v, o)), t2)
    ints = ints_dict(inp)
    s = Solver(o, v, slices=(2, 2, 2), autotune=False, **kw)
    if method == "standard":
        s.set_inputs(eps_o, eps_v, **ints)
    elif method == "df":
        s.set_df_inputs(eps_o, eps_v, np.ascontiguousarray(B[:, o:, :o]), np.ascontiguousarray(B[:, o:, o:]),
                        **{k: ints[k] for k in FOUR})
    else:
        Gao = np.ascontiguousarray(np.einsum("Kpq,Krs->pqrs", Bao, Bao, optimize=True))
        s.set_direct_inputs(eps_o, eps_v, Gao, np.ascontiguousarray(Cm[:, o:]), np.ascontiguousarray(Cm[:, :o]),
                            **{k: ints[k] for k in FOUR + ("Giabc",)})
    return s, inp.t1, inp.t2


def lanes_of(s):
    n, b = C.c_int(), C.c_int64()
    assert s.lib.gbcc_testing_lanes(s.h, C.byref(n), C.byref(b)) == 0
    return n.value, b.value


@pytest.fixture
def hooks():
    lib = _lib.load()
    yield lib
    lib.gbcc_testing_lanes_mode(-1)
    lib.gbcc_testing_free_bytes(-1)
    lib.gbcc_testing_fail_alloc(-1, None)


@pytest.mark.parametrize("o,v", [(1, 1), (3, 8), (11, 46), (24, 90)])
@pytest.mark.parametrize("precision", ["fp64", "mixed", "fp64_tc"])
@pytest.mark.parametrize("method", ["standard", "df", "direct"])
def test_lanes_change_no_bits(hooks, method, precision, o, v):
    if precision == "fp64" and o > 20:
        o, v = 16, 60
    hooks.gbcc_testing_lanes_mode(0)
    s, t1, t2 = make(method, o, v, precision=precision, use_graphs=1)
    with s:
        assert lanes_of(s)[0] == 1
        ref = s.residual(t1, t2)
    hooks.gbcc_testing_lanes_mode(1)
    for graphs in (0, 1):
        s, t1, t2 = make(method, o, v, precision=precision, use_graphs=graphs)
        with s:
            assert lanes_of(s)[0] == 4
            for _ in range(4):
                got = s.residual(t1, t2)
                assert np.array_equal(got[0], ref[0]) and np.array_equal(got[1], ref[1])


@pytest.mark.parametrize("precision", ["fp64", "mixed", "fp64_tc"])
def test_one_lane_where_memory_is_short(hooks, precision):
    got = {}
    for mode, free in ((0, -1), (1, -1), (-1, 0), (-1, 1 << 40)):
        hooks.gbcc_testing_lanes_mode(mode)
        hooks.gbcc_testing_free_bytes(free)
        s, t1, t2 = make("standard", 6, 24, precision=precision)
        with s:
            got[mode, free] = lanes_of(s)
            s.residual(t1, t2)
    assert got[-1, 0] == got[0, -1] and got[0, -1][0] == 1
    assert got[-1, 1 << 40] == got[1, -1] and got[1, -1][0] == 4
    assert got[0, -1][1] < got[1, -1][1]


def test_triples_take_the_workspaces_when_memory_is_short(hooks):
    s, t1, t2 = make("standard", 5, 19, precision="fp64_tc", use_graphs=1)
    with s:
        ref = s.residual(t1, t2)
        for precision in ("mixed", "fp64_tc", "fp64"):
            e = s.triples(precision, t1, t2)
            assert hooks.gbcc_testing_fail_alloc(0, None) == 0  # one allocation of (T) fails
            assert s.triples(precision, t1, t2) == e
            # with the workspaces gone there is nothing left to give
            assert hooks.gbcc_testing_fail_alloc(0, None) == 0
            with pytest.raises(GbccError) as ex:
                s.triples(precision, t1, t2)
            assert ex.value.status == GBCC_ERR_OOM
            got = s.residual(t1, t2)
            assert np.array_equal(got[0], ref[0]) and np.array_equal(got[1], ref[1])


def test_refill_takes_the_workspaces_when_memory_is_short(hooks):
    inp = synth.make_inputs(5, 19, 20, seed=4, t1_scale=1e-2)
    with Solver(5, 19, precision="mixed", slices=(2, 2, 2), autotune=False) as s:
        s.set_inputs(inp.eps_o, inp.eps_v, **ints_dict(inp))
        ref = s.residual(inp.t1, inp.t2)
        assert hooks.gbcc_testing_fail_alloc(0, None) == 0  # (ab|cd), the refill's first allocation
        s.set_inputs(inp.eps_o, inp.eps_v, **ints_dict(inp))
        got = s.residual(inp.t1, inp.t2)
    assert np.array_equal(got[0], ref[0]) and np.array_equal(got[1], ref[1])


def test_packs_of_another_precision_take_the_lanes_when_memory_is_short(hooks):
    s, t1, t2 = make("standard", 13, 57, precision="fp64", use_graphs=1)
    with s:
        ref64 = s.residual(t1, t2)
        ref = s.residual(t1, t2, precision="mixed")
        assert lanes_of(s)[0] == 4
    s, t1, t2 = make("standard", 13, 57, precision="fp64", use_graphs=1)
    with s:
        s.residual(t1, t2)
        assert hooks.gbcc_testing_fail_alloc(1, None) == 0  # the second pack of the mixed plan
        got = s.residual(t1, t2, precision="mixed")
        assert lanes_of(s)[0] == 1
        assert np.array_equal(got[0], ref[0]) and np.array_equal(got[1], ref[1])
        got = s.residual(t1, t2)
        assert np.array_equal(got[0], ref64[0]) and np.array_equal(got[1], ref64[1])
