"""Amplitudes that are not pair-symmetric are refused before anything is done for
their residual: no operand is packed, no pass is run, and what is wrong with them
is reported, not what would have failed on the way."""
import ctypes as C

import numpy as np
import pytest

from conftest import ints_dict
from mpqc_gb300 import Solver, _lib, synth
from mpqc_gb300._lib import GBCC_ERR_INVALID_ARG, GbccError

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("use_graphs", [0, 2])
def test_refused_before_the_residual(use_graphs):
    lib = _lib.load()
    inp = synth.make_inputs(13, 57, 16, seed=2, t1_scale=1e-2)  # packs for the tensor cores
    bad = inp.t2.copy()
    bad[0, 1, 2, 3] += 1.0
    n0, n1 = C.c_int(), C.c_int()
    with Solver(inp.o, inp.v, precision="fp64", use_graphs=use_graphs) as s:
        s.set_inputs(inp.eps_o, inp.eps_v, **ints_dict(inp))
        ref = s.residual(inp.t1, inp.t2)
        assert lib.gbcc_testing_last_launches(s.h, C.byref(n0)) == 0
        out = np.full_like(inp.t1, 7.0), np.full_like(inp.t2, 7.0)
        try:
            # the first mixed residual would pack its operands: that allocation fails
            lib.gbcc_testing_fail_alloc(0, None)
            with pytest.raises(GbccError) as ex:
                s.residual(inp.t1, bad, *out, precision="mixed")
        finally:
            lib.gbcc_testing_fail_alloc(-1, None)
        assert ex.value.status == GBCC_ERR_INVALID_ARG and "pair-symmetric" in str(ex.value)
        assert lib.gbcc_testing_last_launches(s.h, C.byref(n1)) == 0 and n1.value == n0.value
        assert np.all(out[0] == 7.0) and np.all(out[1] == 7.0)
        got = s.residual(inp.t1, inp.t2)
        assert np.array_equal(got[0], ref[0]) and np.array_equal(got[1], ref[1])
