"""Performance cases of the CCSD solver: the calls a user's program makes, over
the sizes it makes them at.

``listed()`` gives fixed cases, ``draw(rng)`` one more case of the same ranges.
``prepare(case, seed)`` builds what the program holds before the call (a
handle with its integrals, the amplitudes), ``run(state)`` makes the call,
``work(case)`` counts the bytes and operations of one call, and
``exact(case, seed)`` gives what the call returns as plain torch FP64
evaluates it.

Inputs are seeded density-fitted integrals over the full orbital space (as in
``mpqc_gb300.synth``, drawn on the GPU), canonical Fock matrices, MP2 doubles
and small random singles: what an amplitude iteration of a closed-shell
molecule meets.  The RHF cases take water clusters whose orientations come
from the seed.

A split-BF16 ("mixed") residual is good to five or six digits
(``slice_tolerance`` is 1e-5), and the program keeps it, as its history of
error vectors, in single precision; FP64 and FP64-grade residuals stay double.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import mpqc_gb300
from mpqc_gb300 import molecules

DEV = "cuda"
BLOCKS = ("Fia", "Fij", "Fab", "Gijab", "Gijkl", "Giajb", "Gijka", "Giabc", "Gabcd")


def listed():
    return [
        # the convergence test of a host-driven amplitude loop on a single
        # water in cc-pVDZ: the smallest call, all latency
        dict(name="energy o5 v19", kind="energy", o=5, v=19, precision="fp64"),
        # a whole default-precision CCSD of that water
        dict(name="solve fp64 o5 v19", kind="solve", o=5, v=19, precision="fp64"),
        # many small molecules at once: water monomers to trimers in 6-31G**,
        # mixed precision with FP64-grade refinement
        dict(name="batch of 6", kind="batch", count=6, largest=3, precision="mixed"),
        # residuals of a host program's own amplitude loop: a ragged small
        # molecule, (H2O)6 / 6-31G** and (H2O)10 / cc-pVDZ, the largest
        dict(name="residual mixed o13 v57", kind="residual", method="standard", o=13, v=57, precision="mixed"),
        dict(name="residual mixed o30 v120", kind="residual", method="standard", o=30, v=120, precision="mixed"),
        dict(name="residual mixed o50 v190", kind="residual", method="standard", o=50, v=190, precision="mixed"),
        # the FP64-grade residual that ends a mixed solve, (H2O)4-sized, ragged
        dict(name="residual fp64_tc o21 v83", kind="residual", method="standard", o=21, v=83, precision="fp64_tc"),
        # density-fitted residual ((ab|cd) never stored), ragged
        dict(name="residual df o24 v131", kind="residual", method="df", o=24, v=131, naux=420, precision="mixed"),
        # integral-direct residual of (H2O)4 / 6-31G**, frozen core
        dict(name="residual direct o16 v80", kind="residual", method="direct", o=16, v=80, nao=100,
             precision="mixed"),
        # (T): (H2O)4 / cc-pVDZ in mixed precision, a smaller ragged one FP64-grade
        dict(name="triples mixed o20 v76", kind="triples", o=20, v=76, precision="mixed"),
        dict(name="triples fp64_tc o12 v51", kind="triples", o=12, v=51, precision="fp64_tc"),
        # the input producer: integrals and RHF of (H2O)4 / 6-31G**
        dict(name="rhf 4 waters", kind="rhf", waters=4, basis="6-31G**"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["energy", "solve", "batch", "mixed", "mixed", "mixed", "fp64", "fp64_tc", "df", "direct",
                       "triples", "triples", "rhf"])

    def ov(lo, hi):
        v = _log_int(rng, lo, hi)
        return dict(o=max(2, int(v * rng.uniform(0.16, 0.27))), v=v)

    if kind == "energy":
        return dict(kind="energy", precision="fp64", **ov(8, 150))
    if kind == "solve":
        return dict(kind="solve", precision=rng.choice(["fp64", "fp64_tc"]), **ov(8, 30))
    if kind == "batch":
        return dict(kind="batch", count=rng.randrange(2, 8), largest=rng.randrange(1, 4), precision="mixed")
    if kind == "mixed":
        return dict(kind="residual", method="standard", precision="mixed", **ov(19, 185))
    if kind == "fp64":
        return dict(kind="residual", method="standard", precision="fp64", **ov(10, 60))
    if kind == "fp64_tc":
        return dict(kind="residual", method="standard", precision="fp64_tc", **ov(19, 110))
    if kind == "df":
        d = ov(30, 140)
        return dict(kind="residual", method="df", precision="mixed", naux=int(d["v"] * rng.uniform(2.5, 4.0)), **d)
    if kind == "direct":
        d = ov(19, 90)
        return dict(kind="residual", method="direct", precision="mixed", nao=d["o"] + d["v"] + rng.randrange(0, 6), **d)
    if kind == "triples":
        prec = rng.choice(["mixed", "mixed", "fp64_tc", "fp64"])
        return dict(kind="triples", precision=prec, **(ov(12, 80) if prec == "mixed" else ov(12, 52)))
    return dict(kind="rhf", waters=rng.randrange(1, 5), basis=rng.choice(["6-31G", "6-31G**", "cc-pVDZ"]))


# ---------------------------------------------------------------------------
# inputs


def _generator(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _square(X):
    """X^T X with exactly symmetric elements; FP32 products above 4 GB of result."""
    n = X.shape[1]
    if n * n > 1 << 29:
        M = (X.float().T @ X.float()).double()
    else:
        M = X.T @ X
    T = M.T.contiguous()
    M += T
    M *= 0.5
    return M


def _product(X, Y):
    """X^T Y (FP32 products above 4 GB of result)."""
    if X.shape[1] * Y.shape[1] > 1 << 29:
        return (X.float().T @ Y.float()).double()
    return X.T @ Y


def _orbital_factor(gen, n, naux, v):
    """A symmetric factor B[Q,p,q] whose integrals have a standard deviation of 0.15 / v."""
    b = math.sqrt(0.15 / v / math.sqrt(naux))
    x = torch.randn(naux, n, n, dtype=torch.float64, device=DEV, generator=gen)
    return (x + x.transpose(1, 2)) * (b * 0.5 ** 0.5)


def _blocks(B, o, names=BLOCKS):
    """The <pq|rs> = (pr|qs) blocks of a factor over the full orbital space."""
    n = B.shape[1]
    v, q = n - o, B.shape[0]
    oo = B[:, :o, :o].reshape(q, -1)
    ov = B[:, :o, o:].reshape(q, -1)
    vv = B[:, o:, o:].reshape(q, -1)
    make = {
        "Gijab": lambda: _square(ov).view(o, v, o, v).permute(0, 2, 1, 3),
        "Gijkl": lambda: _square(oo).view(o, o, o, o).permute(0, 2, 1, 3),
        "Giajb": lambda: _product(oo, vv).view(o, o, v, v).permute(0, 2, 1, 3),
        "Gijka": lambda: _product(oo, ov).view(o, o, o, v).permute(0, 2, 1, 3),
        "Giabc": lambda: _product(ov, vv).view(o, v, v, v).permute(0, 2, 1, 3),
        "Gabcd": lambda: _square(vv).view(v, v, v, v).permute(0, 2, 1, 3),
    }
    return {k: make[k]().contiguous() for k in names if k in make}


def _system(case, seed):
    """Orbital energies, integrals (as the method takes them) and amplitudes."""
    o, v = case["o"], case["v"]
    method = case.get("method", "standard")
    gen = _generator(seed)
    d = {}
    eps_o = torch.sort(torch.rand(o, dtype=torch.float64, device=DEV, generator=gen) * 1.2 - 1.5).values
    eps_v = torch.sort(torch.rand(v, dtype=torch.float64, device=DEV, generator=gen) * 2.9 + 0.1).values
    if method == "direct":
        # AO factor and orthonormal orbitals; the MO factor is its transform
        n = case["nao"]
        B = _orbital_factor(gen, n, 2 * n, v)
        C = torch.linalg.qr(torch.randn(n, n, dtype=torch.float64, device=DEV, generator=gen)).Q
        d["Gao"] = _square(B.reshape(B.shape[0], -1)).view(n, n, n, n)
        C = C[:, n - o - v:].contiguous()
        d["Ci"], d["Ca"] = C[:, :o].contiguous(), C[:, o:].contiguous()
        B = torch.einsum("pi,Qpq,qj->Qij", C, B, C)
        names = tuple(k for k in BLOCKS if k != "Gabcd")
    elif method == "df":
        B = _orbital_factor(gen, o + v, case["naux"], v)
        d["Xai"] = B[:, o:, :o].contiguous()
        d["Xab"] = B[:, o:, o:].contiguous()
        names = tuple(k for k in BLOCKS if k not in ("Giabc", "Gabcd"))
    else:
        B = _orbital_factor(gen, o + v, 2 * (o + v), v)
        names = BLOCKS
    d.update(_blocks(B, o, names))
    d["Fia"] = torch.zeros(o, v, dtype=torch.float64, device=DEV)
    d["Fij"], d["Fab"] = torch.diag(eps_o), torch.diag(eps_v)
    t1 = 1e-2 * torch.randn(v, o, dtype=torch.float64, device=DEV, generator=gen)
    den = (eps_o[None, :] + eps_o[:, None])[None, None] - (eps_v[None, :] + eps_v[:, None])[:, :, None, None]
    t2 = d["Gijab"].permute(2, 3, 0, 1) / den
    t2 = (0.5 * (t2 + t2.permute(1, 0, 3, 2))).contiguous()
    return eps_o, eps_v, d, t1, t2, B


def _residuals_near_convergence(seed, t1, t2):
    gen = _generator(seed + 1)
    r1 = 1e-4 * torch.randn(*t1.shape, dtype=torch.float64, device=DEV, generator=gen)
    r2 = 1e-4 * torch.randn(*t2.shape, dtype=torch.float64, device=DEV, generator=gen)
    return r1, (0.5 * (r2 + r2.permute(1, 0, 3, 2))).contiguous()


def _handle(case, eps_o, eps_v, ints, **kw):
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    s = mpqc_gb300.Solver(case["o"], case["v"], precision=case["precision"], **kw)
    method = case.get("method", "standard")
    ints = dict(ints)
    if method == "df":
        s.set_df_inputs(eps_o, eps_v, ints.pop("Xai"), ints.pop("Xab"), **ints)
    elif method == "direct":
        s.set_direct_inputs(eps_o, eps_v, ints.pop("Gao"), ints.pop("Ca"), ints.pop("Ci"), **ints)
    else:
        s.set_inputs(eps_o, eps_v, **ints)
    return s


def _batch_members(case):
    """Water clusters of 1..largest molecules in 6-31G**, in turn."""
    return [dict(kind="solve", o=5 * n, v=20 * n, precision=case["precision"])
            for n in (1 + k % case["largest"] for k in range(case["count"]))]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "rhf":
        sym, xyz = molecules.water_cluster(case["waters"], seed=seed)
        # distorted a little by the seed: rotations alone leave a monomer as it is
        xyz = xyz + np.random.default_rng(seed).normal(0.0, 0.01, xyz.shape)
        return dict(case=case, symbols=sym, coords=xyz)
    if kind == "batch":
        solvers = []
        for k, m in enumerate(_batch_members(case)):
            eo, ev, d, _, _, B = _system(m, 1000 * seed + k)
            del B
            solvers.append(_handle(m, eo, ev, d, target_precision=1e-8, max_iter=60, refine_precision="fp64_tc",
                                   autotune=False))
        torch.cuda.empty_cache()
        return dict(case=case, solvers=solvers)
    eo, ev, d, t1, t2, B = _system(case, seed)
    del B
    # (T) runs from an FP64 handle in its own precision, as after a solve
    kw = dict(max_iter=60, target_precision=1e-9) if kind == "solve" else {}
    m = dict(case, precision="fp64_tc" if case["precision"] == "fp64_tc" else "fp64") if kind == "triples" else case
    s = _handle(m, eo, ev, d, **kw)
    st = dict(case=case, solver=s, t1=t1, t2=t2)
    if kind == "energy":
        st["r1"], st["r2"] = _residuals_near_convergence(seed, t1, t2)
    if kind == "residual":
        st["r1"], st["r2"] = torch.empty_like(t1), torch.empty_like(t2)
    del d
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return st


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "rhf":
        with mpqc_gb300.RHF(state["symbols"], state["coords"], case["basis"], threshold=1e-11, max_iter=60) as scf:
            e = scf.run()
            _, eps = scf.orbitals()
        return dict(energy=e, eps=eps)
    if kind == "batch":
        return [e for e, _ in mpqc_gb300.solve_batch(state["solvers"])]
    s = state["solver"]
    if kind == "solve":
        e, t1, t2, _ = s.solve()
        return dict(energy=e, t1=t1, t2=t2)
    # the library works on a stream of its own: what torch still has to do on
    # these arrays comes first
    torch.cuda.current_stream().synchronize()
    if kind == "energy":
        e, err = s.energy(state["t1"], state["t2"], state["r1"], state["r2"])
        return dict(energy=e, error=err)
    if kind == "triples":
        return s.triples(case["precision"], state["t1"], state["t2"])
    r1, r2 = s.residual(state["t1"], state["t2"], state["r1"], state["r2"])
    if case["precision"] == "mixed":
        return dict(r1=r1.float(), r2=r2.float())
    return dict(r1=r1, r2=r2)


# ---------------------------------------------------------------------------
# work


def _residual_work(case):
    o, v = float(case["o"]), float(case["v"])
    method = case.get("method", "standard")
    words = 4 * o**2 * v**2 + o**3 * v + o**4
    # ladder over pairs of virtuals and of occupieds, four ring products, the
    # hole-hole ladder, the singles terms
    flops = 9 * o**3 * v**3 + o**4 * v**2 + 14 * o**2 * v**3
    if method == "df":
        words += case["naux"] * v * (v + o)
        flops += 0.5 * o**2 * v**4 + case["naux"] * v**4
    elif method == "direct":
        words += float(case["nao"])**4 + o * v**3
        flops += 0.5 * o**2 * float(case["nao"])**4
    else:
        words += v**4 + o * v**3
        flops += 0.5 * o**2 * v**4
    return 8 * words, flops


def work(case):
    kind = case["kind"]
    if kind == "rhf":
        # basis functions of one water; every unique integral formed (some
        # fifty operations at least), then read by about ten Fock builds
        n = case["waters"] * {"6-31G": 13, "6-31G**": 25, "cc-pVDZ": 24}[case["basis"]]
        return dict(bytes=8.0 * 3 * n * n, flops=n**4 / 8 * (50 + 10 * 8))
    if kind == "batch":
        parts = [work(m) for m in _batch_members(case)]
        return dict(bytes=sum(p["bytes"] for p in parts), flops=sum(p["flops"] for p in parts))
    o, v = float(case["o"]), float(case["v"])
    if kind == "energy":
        return dict(bytes=8.0 * (3 * o**2 * v**2 + 3 * o * v), flops=6 * o**2 * v**2)
    if kind == "triples":
        triplets = o * (o + 1) * (o + 2) / 6
        return dict(bytes=8.0 * (o * v**3 + 2 * o**2 * v**2 + o**3 * v), flops=triplets * 12 * v**3 * (v + o))
    b, f = _residual_work(case)
    if kind == "solve":
        return dict(bytes=b, flops=15 * f)  # some fifteen iterations
    return dict(bytes=b, flops=f)


# ---------------------------------------------------------------------------
# the same results in plain torch FP64


def _residual64(I, t1, t2):
    """Closed-shell CCSD singles and doubles residuals (spin-adapted, canonical
    integrals I)."""
    es = torch.einsum
    Fia, Gijab, Gijka, Giabc, Giajb = I["Fia"], I["Gijab"], I["Gijka"], I["Giabc"], I["Giajb"]
    tau = t2 + es("ai,bj->abij", t1, t1)
    gbar = 2 * Gijab - Gijab.permute(1, 0, 2, 3)
    Fvv = I["Fab"] - es("klcd,adkl->ac", gbar, tau)
    Foo = I["Fij"] + es("klab,abil->ki", gbar, tau)
    Fov = Fia + es("klcd,dl->kc", gbar, t1)
    r1 = Fia.T - 2 * (t1 @ (Fia @ t1)) + Fvv @ t1 - t1 @ Foo
    r1 = r1 + es("kc,caki->ai", Fov, 2 * t2 - t2.permute(0, 1, 3, 2)) + t1 @ (Fov @ t1)
    r1 = r1 + 2 * es("kica,ck->ai", Gijab, t1) - es("kaic,ck->ai", Giajb, t1)
    X = es("kacd,cdij->kaij", Giabc, tau)
    r1 = r1 + 2 * es("kaki->ai", X) - es("kaik->ai", X)
    gooov = 2 * Gijka - Gijka.permute(1, 0, 2, 3)
    r1 = r1 - es("lkic,cakl->ai", gooov, tau)

    r2 = es("icab,cj->abij", Giabc, t1)
    r2 = r2 - es("kbij,ak->abij", es("kbic,cj->kbij", Giajb, t1), t1)
    r2 = r2 - es("jika,bk->abij", Gijka, t1)
    r2 = r2 - es("ikaj,bk->abij", es("ikac,cj->ikaj", Gijab, t1), t1)
    Goo = Foo + Fia @ t1 + es("klic,cl->ki", gooov, t1)
    Gvv = Fvv + t1 @ Fia + 2 * es("kadc,dk->ac", Giabc, t1) - es("kacd,dk->ac", Giabc, t1)
    r2 = r2 + es("ac,cbij->abij", Gvv, t2) - es("ki,abkj->abij", Goo, t2)
    T = 0.5 * t2 + es("di,al->dail", t1, t1)
    J = Gijab.permute(2, 1, 0, 3) - es("lkic,al->akic", Gijka, t1) + es("kacd,di->akic", Giabc, t1)
    J = J - es("klcd,dail->akic", Gijab, T)
    J = J + 0.5 * es("klcd,adil->akic", 2 * Gijab - Gijab.permute(0, 1, 3, 2), t2)
    K = Giajb - es("klic,al->kaic", Gijka, t1) + es("kadc,di->kaic", Giabc, t1) - es("kldc,dail->kaic", Gijab, T)
    r2 = r2 + 0.5 * es("akic,cbkj->abij", 2 * J - K.permute(1, 0, 2, 3), 2 * t2 - t2.permute(1, 0, 2, 3))
    Z = es("kaic,cbjk->abij", K, t2)
    r2 = r2 - 0.5 * Z - Z.permute(1, 0, 2, 3)
    r2 = r2 + r2.permute(1, 0, 3, 2) + Gijab.permute(2, 3, 0, 1)
    W = I["Gijkl"] + es("klic,cj->klij", Gijka, t1) + es("lkjc,ci->klij", Gijka, t1) + es("klcd,cdij->klij", Gijab, tau)
    r2 = r2 + es("klij,abkl->abij", W, tau)
    r2 = r2 + es("abcd,cdij->abij", I["Gabcd"], tau)
    r2 = r2 - es("kaji,bk->abij", X, t1) - es("kbij,ak->abij", X, t1)
    return r1, r2


def _energy64(I, t1, t2, r1, r2):
    """Correlation energy with the residuals added to the integrals."""
    tau = t2 + torch.einsum("ai,bj->abij", t1, t1)
    g = I["Gijab"].permute(2, 3, 0, 1)
    return 2 * torch.sum((I["Fia"].T + r1) * t1) + torch.sum((g + r2) * (2 * tau - tau.permute(1, 0, 2, 3)))


def _solve64(I, eps_o, eps_v):
    """Converged amplitudes and energy by Jacobi steps with DIIS."""
    d1 = eps_o[None, :] - eps_v[:, None]
    d2 = (eps_o[None, :] + eps_o[:, None])[None, None] - (eps_v[None, :] + eps_v[:, None])[:, :, None, None]
    t1, t2 = torch.zeros_like(d1), (I["Gijab"].permute(2, 3, 0, 1) / d2).contiguous()
    xs, rs = [], []
    for _ in range(80):
        r1, r2 = _residual64(I, t1, t2)
        s1, s2 = r1 / d1, r2 / d2
        step = torch.cat([s1.reshape(-1), s2.reshape(-1)])
        xs.append(torch.cat([t1.reshape(-1), t2.reshape(-1)]) + step)
        rs.append(step)
        if step.norm() < 1e-13:
            break
        xs, rs = xs[-8:], rs[-8:]
        n = len(rs)
        R = torch.stack(rs)
        M = torch.ones(n + 1, n + 1, dtype=torch.float64, device=DEV)
        G = R @ R.T
        M[:n, :n] = G / G[-1, -1]
        M[n, n] = 0
        rhs = torch.zeros(n + 1, dtype=torch.float64, device=DEV)
        rhs[n] = 1
        c = torch.linalg.lstsq(M.cpu(), rhs.cpu()[:, None], driver="gelsd").solution[:n, 0].to(DEV)
        x = c @ torch.stack(xs)
        t1, t2 = x[:t1.numel()].view_as(t1), x[t1.numel():].view_as(t2)
    z1, z2 = torch.zeros_like(t1), torch.zeros_like(t2)
    return _energy64(I, t1, t2, z1, z2), t1, t2


def _triples64(I, eps_o, eps_v, t1, t2):
    """The connected and disconnected triples energy, over i <= j <= k."""
    o, v = len(eps_o), len(eps_v)
    es = torch.einsum
    G, R, g = I["Giabc"], I["Gijka"], I["Gijab"]
    t2o = t2.permute(2, 3, 0, 1).contiguous()  # [i][j][a][b]
    dv = eps_v[:, None, None] + eps_v[None, :, None] + eps_v[None, None, :]
    total = torch.zeros((), dtype=torch.float64, device=DEV)
    for i in range(o):
        for j in range(i, o):
            k = slice(j, o)
            # X(x,y,z)[p,q,r] = sum_d <xd|pq> t2(d,r,y,z) - sum_l <yz|lr> t2(p,q,x,l), k batched first
            W = es("dpq,kdr->kpqr", G[i], t2o[j, k]) - es("klr,lpq->kpqr", R[j, k], t2o[i])
            W = W + (es("dpq,kdr->kpqr", G[i], t2o[k, j])
                     - es("klr,lpq->kpqr", R[k, j], t2o[i])).permute(0, 1, 3, 2)
            W = W + (es("dpq,kdr->kpqr", G[j], t2o[i, k])
                     - es("klr,lpq->kpqr", R[i, k], t2o[j])).permute(0, 2, 1, 3)
            W = W + (es("dpq,kdr->kpqr", G[j], t2o[k, i])
                     - es("klr,lpq->kpqr", R[k, i], t2o[j])).permute(0, 3, 1, 2)
            W = W + (es("kdpq,dr->kpqr", G[k], t2o[i, j])
                     - es("lr,klpq->kpqr", R[i, j], t2o[k])).permute(0, 2, 3, 1)
            W = W + (es("kdpq,dr->kpqr", G[k], t2o[j, i])
                     - es("lr,klpq->kpqr", R[j, i], t2o[k])).permute(0, 3, 2, 1)
            V = (es("ab,ck->kabc", g[i, j], t1[:, k]) + es("kbc,a->kabc", g[j, k], t1[:, i])
                 + es("kac,b->kabc", g[i, k], t1[:, j]))
            Y = (4 * W + W.permute(0, 2, 3, 1) + W.permute(0, 3, 1, 2)
                 - 2 * (W.permute(0, 3, 2, 1) + W.permute(0, 1, 3, 2) + W.permute(0, 2, 1, 3)))
            den = (eps_o[i] + eps_o[j] + eps_o[k])[:, None, None, None] - dv
            e = ((W + V) * Y / den).sum(dim=(1, 2, 3))
            mult = torch.full((o - j,), 6.0 if i < j else 3.0, dtype=torch.float64, device=DEV)
            mult[0] = 1.0 if i == j else 3.0  # k = j
            total = total + (mult * e).sum()
    return total / 3


def exact(case, seed):
    kind = case["kind"]
    if kind == "rhf":
        return None
    if kind == "batch":
        out = []
        for k, m in enumerate(_batch_members(case)):
            eo, ev, d, _, _, _ = _system(m, 1000 * seed + k)
            out.append(float(_solve64(d, eo, ev)[0]))
        return out
    eo, ev, d, t1, t2, B = _system(case, seed)
    if kind == "solve":
        e, t1, t2 = _solve64(d, eo, ev)
        return dict(energy=float(e), t1=t1, t2=t2)
    if kind == "energy":
        r1, r2 = _residuals_near_convergence(seed, t1, t2)
        n = t1.numel() + t2.numel()
        return dict(energy=float(_energy64(d, t1, t2, r1, r2)),
                    error=float(torch.sqrt(r1.square().sum() + r2.square().sum()) / n))
    if kind == "triples":
        return float(_triples64(d, eo, ev, t1, t2))
    if work(case)["flops"] > 2e13:
        return None  # some twenty seconds of FP64
    if "Gabcd" not in d:
        names = ("Gabcd",) if "Giabc" in d else ("Giabc", "Gabcd")
        d.update(_blocks(B, case["o"], names))
    del B
    r1, r2 = _residual64(d, t1, t2)
    return dict(r1=r1, r2=r2)
