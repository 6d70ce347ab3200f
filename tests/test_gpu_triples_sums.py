"""The energy sums of (T) in mixed precision on integers: contractions, terms and
denominators that FP32 holds exactly, so that E(T) is exact unless the terms of
the six orderings of a set {a, b, c}, the denominators or the running sum are
formed in FP32 alone."""
import numpy as np
import pytest

from mpqc_gb300 import Solver
from oracle import ccsd_t_ref as T

pytestmark = pytest.mark.gpu


def integer_inputs(o, v, seed):
    rng = np.random.default_rng(seed)
    t1 = rng.choice([-35.0, 35.0], size=(v, o))
    t2 = rng.integers(-4, 5, size=(v, v, o, o)).astype(np.float64)
    t2 = t2 + t2.transpose(1, 0, 3, 2)
    Gijab = rng.choice([-41.0, -40.0, 40.0, 41.0], size=(o, o, v, v))
    Gijka = rng.integers(-3, 4, size=(o, o, o, v)).astype(np.float64)
    Giabc = rng.integers(-3, 4, size=(o, v, v, v)).astype(np.float64)
    return t1, t2, Gijab, Gijka, Giabc


def terms(t1, t2, Gijab, Gijka, Giabc, i, j, k):
    """The integers (W + V) (4 W + ...) of one triplet over [a][b][c]."""
    W, V = T.triplet_blocks(t1, t2, Gijab, Gijka, Giabc, i, j, k)
    y = 4.0 * W + W.transpose(2, 0, 1) + W.transpose(1, 2, 0) - 2.0 * (
        W.transpose(2, 1, 0) + W.transpose(0, 2, 1) + W.transpose(1, 0, 2))
    return (W + V) * y


@pytest.mark.parametrize("shift", [0.0, 1000.0 + 5.0 * 2.0 ** -15])
@pytest.mark.parametrize("o,v,seed", [(3, 9, 1), (4, 40, 2)])
def test_mixed_energy_sums_are_exact_on_integers(o, v, seed, shift):
    args = integer_inputs(o, v, seed)
    total, wide = 0.0, 0
    for i in range(o):
        for j in range(i, o):
            for k in range(j, o):
                x = terms(*args, i, j, k)
                assert np.abs(x).max() < 2.0 ** 24  # FP32 holds every term
                six = sum(x.transpose(p) for p in ((0, 1, 2), (1, 2, 0), (2, 0, 1), (2, 1, 0), (0, 2, 1), (1, 0, 2)))
                wide += int(np.sum(np.abs(six) > 2.0 ** 24))
                total += (6.0 if i < j < k else (1.0 if i == j == k else 3.0)) * x.sum()
    assert wide > 100 or v < 40  # and not all sums over the six orderings
    t1, t2, Gijab, Gijka, Giabc = args
    # every denominator is -6; the shift cancels in it
    eps_o, eps_v = np.full(o, shift - 0.75), np.full(v, shift + 1.25)
    z = np.zeros
    with Solver(o, v, precision="fp64") as s:
        s.set_inputs(eps_o, eps_v, Fia=z((o, v)), Fij=np.diag(eps_o), Fab=np.diag(eps_v), Gijab=Gijab,
                     Gijkl=z((o, o, o, o)), Giajb=z((o, v, o, v)), Gijka=Gijka, Giabc=Giabc, Gabcd=z((v, v, v, v)))
        e = s.triples("mixed", t1, t2)
    # an exact sum, its share of -1/6 and the final third
    assert abs(e - total / -6.0 / 3.0) <= 2.0 ** -50 * abs(total)
