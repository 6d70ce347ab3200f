"""(T) on the tensor cores past 2^30 elements of a triplet's sums (v > 1024), from
density-fitted inputs of two occupied orbitals, against the same energy in
plain torch FP64: with a factor of rank 2 the connected triples are sums of outer
products."""
import numpy as np
import pytest

from mpqc_gb300 import Solver

pytestmark = pytest.mark.gpu

O, V, NAUX = 2, 1030, 2
TOL = {"mixed": 2e-5, "fp64_tc": 1e-11}  # as at the other sizes (test_gpu_triples.py)


def _reference(torch, B, t1, t2, R, Gijab, eps_o, eps_v):
    Bov, Bvv = B[:, :O, O:], B[:, O:, O:]

    def x(i, j, k):  # [p,q,r]: sum_d <id|pq> t2(d,r,j,k) - sum_l <jk|lr> t2(p,q,i,l)
        y = torch.einsum("Kdq,dr->Kqr", Bvv, t2[:, :, j, k])
        out = torch.einsum("Kp,Kqr->pqr", Bov[:, i], y)
        for l in range(O):
            out -= t2[:, :, i, l].unsqueeze(2) * R[j, k, l]
        return out

    e = 0.0
    for i, j, k in ((0, 0, 1), (0, 1, 1)):
        W = x(i, j, k)
        W += x(i, k, j).permute(0, 2, 1)
        W += x(j, i, k).permute(1, 0, 2)
        W += x(j, k, i).permute(2, 0, 1)
        W += x(k, i, j).permute(1, 2, 0)
        W += x(k, j, i).permute(2, 1, 0)
        total = 0.0
        for a in range(0, V, 103):
            s = slice(a, a + 103)
            w = W[s]
            y = 4.0 * w + W.permute(1, 2, 0)[s] + W.permute(2, 0, 1)[s] - 2.0 * (
                W.permute(2, 1, 0)[s] + W.permute(0, 2, 1)[s] + W.permute(1, 0, 2)[s])
            y *= w + (Gijab[i, j][s, :, None] * t1[:, k] + Gijab[j, k] * t1[s, None, None, i]
                      + Gijab[i, k][s, None, :] * t1[:, None, j])
            y /= (eps_o[i] + eps_o[j] + eps_o[k] - eps_v[s, None, None] - eps_v[:, None] - eps_v)
            total += float(y.sum())
        e += 3.0 * total  # i <= j <= k with two equal; i = j = k gives nothing
    return e / 3.0


def test_triples_past_a_32_bit_sum_array():
    import torch
    if torch.cuda.mem_get_info()[0] < 240 << 30:
        pytest.skip("needs 240 GB of free device memory")
    g = torch.Generator(device="cuda")
    g.manual_seed(7)

    def rand(*shape):
        return torch.randn(*shape, dtype=torch.float64, device="cuda", generator=g)

    n = O + V
    B = rand(NAUX, n, n) * 0.02
    B = B + B.transpose(1, 2)
    Boo, Bov, Bvv = B[:, :O, :O], B[:, :O, O:], B[:, O:, O:]
    block = lambda p, q: torch.einsum("Kpr,Kqs->pqrs", p, q).contiguous()
    ints = dict(Gijab=block(Bov, Bov), Gijkl=block(Boo, Boo), Giajb=block(Boo, Bvv), Gijka=block(Boo, Bov))
    eps_o = torch.sort(torch.rand(O, dtype=torch.float64, device="cuda", generator=g) - 1.5).values
    eps_v = torch.sort(torch.rand(V, dtype=torch.float64, device="cuda", generator=g) * 2.9 + 0.1).values
    t2 = rand(V, V, O, O) * 1e-2
    t2 = (0.5 * (t2 + t2.permute(1, 0, 3, 2))).contiguous()
    t1 = rand(V, O) * 1e-2
    ref = _reference(torch, B, t1, t2, ints["Gijka"], ints["Gijab"], eps_o, eps_v)
    ints.update(Fia=torch.zeros(O, V, dtype=torch.float64, device="cuda"), Fij=torch.diag(eps_o), Fab=torch.diag(eps_v))
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    with Solver(O, V, precision="fp64") as s:
        s.set_df_inputs(eps_o, eps_v, B[:, O:, :O].contiguous(), Bvv.contiguous(), **ints)
        got = {p: s.triples(p, t1, t2) for p in TOL}
    for p, e in got.items():
        print(f"{p}: E(T) {e:.12e}, torch {ref:.12e}, rel {abs(e - ref) / abs(ref):.2e}")
        assert abs(e - ref) <= TOL[p] * abs(ref)
