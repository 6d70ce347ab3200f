"""The one-launch energy sums (gbcc_energy) against numpy: fewer pairs (a, b) than
reduction blocks and more, host and device arrays, repeated calls (the block
counter returns to zero)."""
import numpy as np
import pytest

from conftest import ints_dict
from mpqc_gb300 import Solver, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("o,v", [(1, 1), (2, 3), (5, 24), (3, 25), (9, 33)])
def test_energy_matches_numpy(o, v):
    import torch
    inp = synth.make_inputs(o, v, 8, seed=o * 100 + v, t1_scale=1e-2)
    rng = np.random.default_rng(v)
    r1, r2 = rng.normal(size=(v, o)), rng.normal(size=(v, v, o, o))
    tau = inp.t2 + np.einsum("ai,bj->abij", inp.t1, inp.t1)
    g = inp.Gijab.transpose(2, 3, 0, 1)
    terms = (g + r2) * (2.0 * tau - tau.transpose(1, 0, 2, 3))
    ref = 2.0 * np.sum((inp.Fia.T + r1) * inp.t1) + np.sum(terms)
    err = np.sqrt(np.sum(r1 * r1) + np.sum(r2 * r2)) / (r1.size + r2.size)
    bound = 2.0 ** -52 * terms.size * (np.sum(np.abs(terms)) + 2.0 * np.sum(np.abs(r1 * inp.t1)))
    host = [np.ascontiguousarray(x) for x in (inp.t1, inp.t2, r1, r2)]
    dev = [torch.from_numpy(x).cuda() for x in host]
    torch.cuda.synchronize()
    with Solver(o, v) as s:
        s.set_inputs(inp.eps_o, inp.eps_v, **ints_dict(inp))
        got = [s.energy(*args) for args in (host, dev, dev, host)]
    assert all(x == got[0] for x in got)
    assert abs(got[0][0] - ref) <= bound and abs(got[0][1] - err) <= 1e-12 * err
