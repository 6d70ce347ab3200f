"""A residual pass that fails on the host midway (an operation that is not
launched): the call reports it, nothing of the pass still runs when it has, and
the handle evaluates the next residual."""
import ctypes as C

import pytest

from conftest import ints_dict, rel_err
from mpqc_gb300 import Solver, _lib, synth
from mpqc_gb300._lib import GBCC_ERR_CUDA, GbccError

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("use_graphs", [0, 1])
@pytest.mark.parametrize("site", [3, 30, 53])
def test_failed_pass_leaves_nothing_running(site, use_graphs):
    lib = _lib.load()
    # plain FP64 at a size whose operations take long enough to still be queued
    # when the failing one is reached
    inp = synth.make_inputs(12, 60, 20, seed=3, t1_scale=1e-2)
    busy = C.c_int(-1)
    with Solver(inp.o, inp.v, precision="fp64", use_graphs=use_graphs) as s:
        s.set_inputs(inp.eps_o, inp.eps_v, **ints_dict(inp))
        try:
            assert lib.gbcc_testing_fail_site(site) == 0
            with pytest.raises(GbccError) as ex:
                s.residual(inp.t1, inp.t2)
            assert lib.gbcc_testing_lanes_busy(s.h, C.byref(busy)) == 0
        finally:
            lib.gbcc_testing_fail_site(-1)
        assert ex.value.status == GBCC_ERR_CUDA and "injected" in str(ex.value)
        assert busy.value == 0
        r1, r2 = s.residual(inp.t1, inp.t2)
    with Solver(inp.o, inp.v, precision="fp64") as s:
        s.set_inputs(inp.eps_o, inp.eps_v, **ints_dict(inp))
        f1, f2 = s.residual(inp.t1, inp.t2)
    assert rel_err(r1, f1) == 0.0 and rel_err(r2, f2) == 0.0
