"""(T) on the tensor cores at the edges of its tiles (8 x 16 virtual pairs, 32 to
128 columns) and of its energy blocks (8 virtuals), against the oracle.
Density-fitted inputs keep (ab|cd) out of the way at the larger sizes."""
import numpy as np
import pytest

from mpqc_gb300 import Solver, synth
from oracle import ccsd_t_ref as T

pytestmark = pytest.mark.gpu

TOL = {"fp64_tc": 1e-11, "mixed": 2e-5}  # as for the whole sizes of test_gpu_triples.py


@pytest.mark.parametrize("precision", ["mixed", "fp64_tc"])
@pytest.mark.parametrize("o,v", [(2, 1), (2, 2), (3, 8), (2, 9), (3, 16), (2, 17), (2, 32), (2, 33), (2, 49), (2, 65),
                                 (2, 81), (2, 97), (2, 113), (2, 129)])
def test_triples_at_tile_edges(o, v, precision):
    rng = np.random.default_rng(100 * o + v)
    B = synth.make_df_factor(rng, 12, o + v, 0.05)
    Boo, Bov, Bvv = B[:, :o, :o], B[:, :o, o:], B[:, o:, o:]

    def g(x, y):
        return np.ascontiguousarray(np.einsum("Qpr,Qqs->pqrs", x, y, optimize=True))

    ints = dict(Fia=np.zeros((o, v)), Gijab=g(Bov, Bov), Gijkl=g(Boo, Boo), Giajb=g(Boo, Bvv), Gijka=g(Boo, Bov))
    eps_o = np.sort(rng.uniform(-1.5, -0.3, size=o))
    eps_v = np.sort(rng.uniform(0.1, 3.0, size=v))
    ints.update(Fij=np.diag(eps_o), Fab=np.diag(eps_v))
    t2 = rng.normal(0.0, 1e-2, size=(v, v, o, o))
    t2 = 0.5 * (t2 + t2.transpose(1, 0, 3, 2))
    t1 = rng.normal(0.0, 1e-2, size=(v, o))
    ref = T.triples_energy_by_triplet(t1, t2, ints["Gijab"], ints["Gijka"], g(Bov, Bvv), eps_o, eps_v)
    with Solver(o, v, precision="fp64") as s:
        s.set_df_inputs(eps_o, eps_v, np.ascontiguousarray(B[:, o:, :o]), np.ascontiguousarray(Bvv), **ints)
        e = s.triples(precision, t1, t2)
    assert abs(e - ref) <= TOL[precision] * abs(ref) + (1e-12 if precision == "mixed" else 1e-16)
