"""Which arrays gbcc_energy reads where they lie, and that the others give the same
sums: device arrays at an odd address or running past their allocation are
copied first, as host arrays are (a copy takes any address and reports a range
it cannot read)."""
import ctypes as C

import numpy as np
import pytest

from conftest import ints_dict
from mpqc_gb300 import Solver, _lib, synth

pytestmark = pytest.mark.gpu


def test_energy_reads_only_what_a_kernel_may_read():
    import torch
    lib = _lib.load()
    host = np.zeros(8)
    # 64 MB: an allocation of torch's own
    t = torch.zeros(1 << 23, dtype=torch.float64, device="cuda")
    at = t.data_ptr()
    assert lib.gbcc_testing_reads_in_place(at, 1 << 23, 0) == 1
    assert lib.gbcc_testing_reads_in_place(at + 8, (1 << 23) - 1, 0) == 1
    assert lib.gbcc_testing_reads_in_place(at + 8, 1 << 30, 0) == 0
    assert lib.gbcc_testing_reads_in_place(at + 8, 1 << 60, 0) == 0
    for k in range(1, 8):
        assert lib.gbcc_testing_reads_in_place(at + k, 8, 0) == 0
    assert lib.gbcc_testing_reads_in_place(host.ctypes.data, 8, 0) == 0
    assert lib.gbcc_testing_reads_in_place(at, 8, 1) == 0


@pytest.mark.parametrize("shift", [0, 1, 4])
def test_energy_of_unaligned_device_arrays(shift):
    import torch
    inp = synth.make_inputs(3, 7, 8, seed=7, t1_scale=1e-2)
    rng = np.random.default_rng(7)
    arrays = [np.ascontiguousarray(x) for x in
              (inp.t1, inp.t2, rng.normal(size=inp.t1.shape), rng.normal(size=inp.t2.shape))]
    raw = []
    for x in arrays:
        b = torch.zeros(x.nbytes + 16, dtype=torch.uint8, device="cuda")
        b[shift:shift + x.nbytes] = torch.from_numpy(x.reshape(-1).view(np.uint8)).cuda()
        raw.append(b)
    torch.cuda.synchronize()
    e, err = C.c_double(), C.c_double()
    with Solver(3, 7) as s:
        s.set_inputs(inp.eps_o, inp.eps_v, **ints_dict(inp))
        ref = s.energy(*arrays)
        assert s.lib.gbcc_energy(s.h, *(b.data_ptr() + shift for b in raw), C.byref(e), C.byref(err)) == 0
    assert (e.value, err.value) == ref
