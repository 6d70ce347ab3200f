"""A solve whose DIIS storage cannot be allocated, twice at different places: each
reports it, and the next solve on the handle is an undisturbed one's."""
import numpy as np
import pytest

from conftest import ints_dict
from mpqc_gb300 import Solver, _lib, synth
from mpqc_gb300._lib import GBCC_ERR_OOM, GbccError

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("places", [(2, 0), (0, 0), (6, 3, 0), (3, 5, 1)])
def test_solve_after_failed_diis_storage(places):
    lib = _lib.load()
    inp = synth.make_inputs(4, 12, 10, seed=11, b_scale=0.02)
    with Solver(inp.o, inp.v, precision="fp64", max_iter=40) as s:
        s.set_inputs(inp.eps_o, inp.eps_v, **ints_dict(inp))
        ref = s.solve()
    with Solver(inp.o, inp.v, precision="fp64", max_iter=40) as s:
        s.set_inputs(inp.eps_o, inp.eps_v, **ints_dict(inp))
        for n in places:
            try:
                assert lib.gbcc_testing_fail_alloc(n, None) == 0
                with pytest.raises(GbccError) as ex:
                    s.solve()
            finally:
                lib.gbcc_testing_fail_alloc(-1, None)
            assert ex.value.status == GBCC_ERR_OOM
        e, t1, t2, rep = s.solve()
    assert e == ref[0] and np.array_equal(t1, ref[1]) and np.array_equal(t2, ref[2])
