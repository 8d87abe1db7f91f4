"""The workloads whose speed is followed: (T) energies and VJPs as a program
that uses this package calls them, over the range of sizes, precision modes
and entry points in use.

A case is a dict of plain values; ``call`` names the entry point:

  energy    triples.energy              E(T) of a whole system
  vjp       triples.energy_vjp          E(T) and every gradient, whole system
  block     ct_energy_vjp_block         one slab block of the driver's loop on
                                        device arrays (the last ``slab`` virtuals)
  lno       triples.lno_energy_vjp      LNO-projected (T) of a fragment, with VJP
  kernel    cc.ccsd_t.kernel            the pyscfad-level call on CUDA tensors in
                                        pyscf layouts, and its backward
  iter      cc.ccsd_t_iter              the iterative 6-D (T) solver to convergence
  df        cc.df                       integrals in kernel layouts from DF
                                        factors, and the factor gradients

Systems follow the recipe of pyscfad_b200/synth.py (orbital energies, ERIs
from a symmetric DF factor, amplitude scales), drawn on the GPU.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from pyscfad_b200 import native, triples
from pyscfad_b200.cc import ccsd_t, ccsd_t_iter, df
from pyscfad_b200.cc.eris import ERIs

KEYS = ("mo_energy", "t1T", "t2T", "vooo", "fvo", "vvop")


# ---------------------------------------------------------------- cases
def listed():
    return [
        # the smallest call: a fragment or test molecule, where the call's own
        # launches and host work are the time
        dict(name="energy_o4v10", call="energy", mode="fp64", o=4, v=10, fvo=0.0),
        # a small molecule's gradient (nocc=8, nvir=40, the first named system)
        dict(name="vjp_o8v40", call="vjp", mode="fp64", o=8, v=40, fvo=0.0),
        # a single-point energy and a gradient of the second named system
        # (nocc=16, nvir=120) in the default precision
        dict(name="energy_o16v120", call="energy", mode="fp64", o=16, v=120, fvo=0.0),
        dict(name="vjp_o16v120", call="vjp", mode="fp64", o=16, v=120, fvo=0.0),
        # odd orbital counts and a non-canonical reference (fvo != 0)
        dict(name="vjp_o23v61_fvo", call="vjp", mode="fp64", o=23, v=61, fvo=0.02),
        # one slab block of a large system, default precision: the unit of work
        # of a long float64 gradient (the benchmark's nocc at a smaller nvir)
        dict(name="block_o48v300", call="block", mode="fp64", o=48, v=300, slab=6, fvo=0.0),
        # the same in TF32 with the benchmark's slab width
        dict(name="block_tf32_o48v300", call="block", mode="tf32", o=48, v=300, slab=24, fvo=0.0),
        # a whole medium system in the split-product mode
        dict(name="vjp_bf16x3_o32v100", call="vjp", mode="bf16x3", o=32, v=100, fvo=0.0),
        # an LNO fragment: projected energy and its VJP
        dict(name="lno_o14v50", call="lno", mode="fp64", o=14, v=50, fvo=0.0),
        # the drop-in call on pyscf-layout tensors with packed ovvv, and backward
        dict(name="kernel_tf32_o16v72", call="kernel", mode="tf32", o=16, v=72, fvo=0.0),
        # non-canonical orbitals solved iteratively
        dict(name="iter_o8v40", call="iter", mode="fp64", o=8, v=40, fvo=0.02),
        # DF integrals of the second named system and their factor gradients
        dict(name="df_o16v120", call="df", mode="fp64", o=16, v=120, fvo=0.0),
    ]


def _n_sorted(v):
    return v * (v + 1) * (v + 2) // 6


def _block_abc(v, slab):
    a0 = v - slab
    return [(a, b, c) for a in range(a0, v) for b in range(a0, a + 1) for c in range(b + 1)]


def _n_jobs(case):
    v = case["v"]
    if case["call"] == "block":
        s = case["slab"]
        return sum(b + 1 for a in range(v - s, v) for b in range(v - s, a + 1))
    return _n_sorted(v)


def _seconds(case):
    """A rough upper estimate of a pass, to keep drawn cases below the largest listed one."""
    w = work(case)
    rate = {"fp64": 18e12, "tf32": 120e12, "bf16x3": 80e12}[case["mode"]]
    t = w["flops"] / rate + w["bytes"] / 3e12
    return t * {"lno": 1.6, "kernel": 1.4, "iter": 4.0}.get(case["call"], 1.0)


def draw(rng):
    while True:
        call = rng.choice(["energy", "energy", "vjp", "vjp", "vjp", "block", "block", "lno", "kernel", "iter", "df"])
        mode = "fp64" if call in ("iter", "df") else rng.choice(["fp64", "fp64", "fp64", "tf32", "bf16x3"])
        o = int(round(math.exp(rng.uniform(math.log(4), math.log(48)))))
        v = int(round(math.exp(rng.uniform(math.log(10), math.log(300)))))
        if mode != "fp64":
            o = max(8, o // 8 * 8)          # the tensor-core modes take multiples of 8
        case = dict(call=call, mode=mode, o=o, v=v, fvo=rng.choice([0.0, 0.0, 0.02]))
        if call == "iter":
            case["fvo"] = 0.02
            if o > 10 or v > 48:
                continue
        if call == "block":
            if v < 60:
                continue
            case["slab"] = rng.randint(3, 24)
        if v < 1.25 * o or 8 * v * v * o * (o + v) > 13e9 or _seconds(case) > 0.45:
            continue
        return case


# ---------------------------------------------------------------- inputs
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 7919 + 17)
    return g


def _factors(case, seed):
    """Orbital energies, the symmetric DF factor B (naux, n, n), t1 and t2 (pyscf layouts), fvo."""
    o, v = case["o"], case["v"]
    n, naux = o + v, 3 * v
    g = _gen(seed)
    kw = dict(dtype=torch.float64, device="cuda", generator=g)
    eo = torch.sort(torch.rand(o, **kw) * 1.7 - 2.0)[0]
    ev = torch.sort(torch.rand(v, **kw) * 2.9 + 0.1)[0]
    X = torch.randn((naux, n, n), **kw)
    B = (X + X.transpose(1, 2)) * (0.5 / math.sqrt(naux))
    del X
    t1 = 1e-4 * torch.randn((o, v), **kw)
    Y = torch.randn((o, o, v, v), **kw)
    t2 = (Y + Y.permute(1, 0, 3, 2)) * 0.5e-2
    del Y
    fvo = case["fvo"] * torch.randn((v, o), **kw)
    return torch.cat([eo, ev]), B, t1, t2, fvo, g


def _layouts(case, seed):
    """The kernel layouts of pyscfad_b200.triples."""
    o, v = case["o"], case["v"]
    n = o + v
    mo, B, t1, t2, fvo, _ = _factors(case, seed)
    naux = B.shape[0]
    Lia = B[:, :o, o:].contiguous()
    R = B[:, :, o:].reshape(naux, n * v)
    vvop = torch.empty((v, v, o, n), dtype=torch.float64, device="cuda")
    for a in range(0, v, 32):
        G = (Lia[:, :, a:a + 32].reshape(naux, -1).t() @ R).view(o, -1, n, v)
        vvop[a:a + 32] = G.permute(1, 3, 0, 2)
    del R, G
    vooo = (Lia.reshape(naux, o * v).t() @ B[:, :o, :o].reshape(naux, o * o)).view(o, v, o, o)
    return dict(mo_energy=mo, t1T=t1.t().contiguous(), t2T=t2.permute(2, 3, 1, 0).contiguous(),
                vooo=vooo.permute(1, 0, 3, 2).contiguous(), fvo=fvo, vvop=vvop)


def _pyscf(case, seed):
    """t1, t2, mo_energy, fock, ovoo, ovov and lower-triangular packed ovvv, as a CC object holds them."""
    o, v = case["o"], case["v"]
    mo, B, t1, t2, fvo, g = _factors(case, seed)
    naux = B.shape[0]
    fock = torch.diag(mo)
    fock[o:, :o] = fvo
    fock[:o, o:] = fvo.t()
    if case["call"] == "iter":
        for lo, hi in ((0, o), (o, o + v)):
            x = 0.02 * torch.randn((hi - lo, hi - lo), dtype=torch.float64, device="cuda", generator=g)
            x = 0.5 * (x + x.t())
            x.diagonal().zero_()
            fock[lo:hi, lo:hi] += x
    Lov = B[:, :o, o:].reshape(naux, -1)
    i, j = np.tril_indices(v)
    i, j = torch.as_tensor(i, device="cuda"), torch.as_tensor(j, device="cuda")
    return dict(t1=t1, t2=t2, mo_energy=mo, fock=fock,
                ovoo=(Lov.t() @ B[:, :o, :o].reshape(naux, -1)).view(o, v, o, o),
                ovov=(Lov.t() @ Lov).view(o, v, o, v),
                ovvv=(Lov.t() @ B[:, o:, o:][:, i, j]).view(o, v, -1))


def _projector(case, seed):
    """mat = u^T u of a fragment's localized occupied orbitals (rank about a third of nocc)."""
    o = case["o"]
    u = torch.randn((max(1, o // 3), o), dtype=torch.float64, device="cuda", generator=_gen(seed + 1))
    u = torch.linalg.qr(u.t())[0].t()
    return (u.t() @ u).contiguous()


def prepare(case, seed):
    call = case["call"]
    if call == "kernel":
        s = {k: x.requires_grad_() for k, x in _pyscf(case, seed).items()}
    elif call == "iter":
        s = _pyscf(case, seed)
    elif call == "df":
        o = case["o"]
        mo, B, t1, t2, fvo, g = _factors(case, seed)
        naux, v = B.shape[0], case["v"]
        i, j = np.tril_indices(v)
        s = dict(t1=t1, t2=t2, mo_energy=mo, fock=torch.diag(mo), Loo=B[:, :o, :o].reshape(naux, -1).contiguous(),
                 Lov=B[:, :o, o:].reshape(naux, -1).contiguous(),
                 Lvv=B[:, o:, o:][:, torch.as_tensor(i, device="cuda"), torch.as_tensor(j, device="cuda")])
        kw = dict(dtype=torch.float64, device="cuda", generator=g)
        s["bars"] = dict(vooo=torch.randn((v, o, o, o), **kw), vvop=torch.randn((v, v, o, o + v), **kw))
    else:
        s = dict(L=_layouts(case, seed))
        if call == "lno":
            s["mat"] = _projector(case, seed)
    s["case"] = dict(case)
    torch.cuda.empty_cache()
    return s


# ---------------------------------------------------------------- one pass
def _ptrs(d):
    return [ctypes.c_void_p(d[k].data_ptr()) for k in KEYS]


def _block(L, mode, v, slab):
    """One diagonal slab block through the C-ABI, as the driver's loop calls it on device arrays."""
    o = L["t1T"].shape[1]
    g = {k: torch.zeros_like(L[k]) for k in KEYS}
    e = torch.zeros((), dtype=torch.float64, device="cuda")
    prob, grads = native.CtProblem(o, v, *_ptrs(L)), native.CtGrads(*_ptrs(g))
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    native.check(native.lib().ct_energy_vjp_block(ctypes.byref(prob), native.mode_id(mode), 2.0, ctypes.byref(grads),
                                                  v - slab, v, v - slab, v, ctypes.c_void_p(e.data_ptr()), st))
    return e, g


def run(state):
    case = state["case"]
    call, mode = case["call"], case["mode"]
    if call == "energy":
        return triples.energy(state["L"], mode=mode)
    if call == "vjp":
        return triples.energy_vjp(state["L"], 2.0, mode=mode)
    if call == "block":
        return _block(state["L"], mode, case["v"], case["slab"])
    if call == "lno":
        return triples.lno_energy_vjp(state["L"], state["mat"], 2.0 / 3.0, mode=mode)
    if call == "df":
        L = df.df_layouts(*[state[k] for k in ("t1", "t2", "mo_energy", "fock", "Loo", "Lov", "Lvv")])
        bars = df.df_factor_bar(state["bars"], state["Loo"], state["Lov"], state["Lvv"])
        return dict(vvop=L["vvop"], vooo=L["vooo"], t2T=L["t2T"], bars=bars)
    eris = ERIs(fock=state["fock"], mo_energy=state["mo_energy"], ovoo=state["ovoo"], ovov=state["ovov"],
                ovvv=state["ovvv"])
    if call == "iter":
        return ccsd_t_iter.iterative_kernel(None, eris, state["t1"], state["t2"])
    x = [state[k] for k in ("t1", "t2", "mo_energy", "fock", "ovoo", "ovov", "ovvv")]
    e = ccsd_t.kernel(None, eris, x[0], x[1], mode=mode)
    return e.detach(), torch.autograd.grad(e, x)


# ---------------------------------------------------------------- what a pass needs
def work(case):
    o, v, call = case["o"], case["v"], case["call"]
    n, naux = o + v, 3 * v
    if call == "df":
        f = 2 * naux * (v * v * o * n + v * o ** 3)
        fac = naux * (o * o + o * v + v * (v + 1) // 2)
        out = v * v * o * n + v * o ** 3
        return {"bytes": 8 * (2 * fac + 2 * out + 4 * (o * v) ** 2), "flops": 3 * f}
    jobs = _n_jobs(case)
    t2, vooo = v * v * o * o, v * o ** 3
    vvop = v * v * o * n
    if call == "block":
        vvop = (v * v - (v - case["slab"]) ** 2) * o * n
    elements = vvop + t2 + vooo + 2 * o * v + n
    flops = 12 * o ** 3 * n * jobs
    if call == "energy":
        return {"bytes": 8 * elements, "flops": flops}
    if call in ("vjp", "block"):
        return {"bytes": 16 * elements, "flops": 3 * flops}
    if call == "lno":
        return {"bytes": 16 * elements, "flops": 3 * flops + 18 * o ** 4 * jobs}
    if call == "kernel":
        packed = o * v * (o * v + o * o + v * (v + 1) // 2) + t2
        return {"bytes": 16 * packed, "flops": 4 * flops}
    # iter: the seed, then a converged solve's Fock products (about ten cycles)
    t3 = (o * v) ** 3
    return {"bytes": 8 * (elements + t3), "flops": flops + 10 * 2 * t3 * n}


# ---------------------------------------------------------------- the same in plain 64-bit torch
R6 = ((0, 1, 2), (0, 2, 1), (1, 0, 2), (1, 2, 0), (2, 0, 1), (2, 1, 0))


def _r3(y):
    """4 y + the two cyclic - 2 x the three exchanged arrangements of the last three axes."""
    p = lambda *q: y.permute(0, *[1 + i for i in q])  # noqa: E731
    return 4 * y + p(1, 2, 0) + p(2, 0, 1) - 2 * (p(2, 1, 0) + p(0, 2, 1) + p(1, 0, 2))


def _triples64(L, abc, weight, cot=None, mat=None):
    """sum_t weight_t sum_ijk (mat^T W)_ijk r3(W + V)_ijk / D_ijk over the virtual
    triples abc (mat: the identity when None), and with ``cot`` the gradients of
    cot x that sum with respect to every input."""
    o, v = L["t1T"].shape[1], L["t1T"].shape[0]
    n = o + v
    dev = L["t1T"].device
    t2z = L["t2T"].view(v, v, o * o)
    vv = L["vvop"].view(v * v, o, n)
    grad = {k: torch.zeros_like(L[k]) for k in KEYS} if cot is not None else None
    mat_bar = torch.zeros_like(mat) if mat is not None and cot is not None else None
    batch = max(1, min(8192, int(2.5e9 / (8 * 6 * (o ** 3 + o * n)) / 3)))
    abc = torch.as_tensor(np.asarray(abc, dtype=np.int64), device=dev)
    weight = torch.as_tensor(np.asarray(weight, dtype=np.float64), device=dev)
    total = torch.zeros((), dtype=torch.float64, device=dev)
    for s in range(0, len(abc), batch):
        J, wt = abc[s:s + batch], weight[s:s + batch]
        nj = len(J)
        xyz = torch.stack([J[:, list(r)] for r in R6])              # (6, nj, 3)
        x, y, z = (xyz[:, :, k].reshape(-1) for k in range(3))
        zs, order = torch.sort(z, stable=True)
        cut = torch.unique_consecutive(zs, return_counts=True)
        zvals, counts = cut[0].tolist(), cut[1].tolist()
        A = vv[x * v + y]                                           # (6 nj, o, n)
        G = torch.empty((6 * nj, o, o * o), dtype=torch.float64, device=dev)
        at = 0
        for zz, cnt in zip(zvals, counts):
            i = order[at:at + cnt]
            G[i] = (A[i, :, o:].reshape(cnt * o, v) @ t2z[zz]).view(cnt, o, o * o)
            at += cnt
        Tzy = L["t2T"][z, y]                                        # (6 nj, l, r)
        Ox = L["vooo"][x].view(6 * nj, o * o, o)
        G = (G.view(6 * nj, o * o, o) - Ox @ Tzy).view(6, nj, o, o, o)
        voo, tyx = A[:, :, :o].contiguous(), L["t2T"][y, x]
        t1z, fz = L["t1T"][z], L["fvo"][z]
        e = L["mo_energy"]
        if cot is not None:
            G, voo, tyx, t1z, fz, e = (q.detach().requires_grad_() for q in (G, voo, tyx, t1z, fz, e))
            m = mat.detach().requires_grad_() if mat is not None else None
        else:
            m = mat
        V = (voo[:, :, :, None] * t1z[:, None, None, :] + tyx[:, :, :, None] * fz[:, None, None, :]).view(6, nj, o, o, o)
        W = Y = 0
        for k, r in enumerate(R6):
            q = (0, *[1 + int(i) for i in np.argsort(r)])
            W = W + G[k].permute(q)
            Y = Y + V[k].permute(q)
        Z = _r3(W + 0.5 * Y)
        D = (e[:o, None, None] + e[None, :o, None] + e[None, None, :o])[None] \
            - e[o + J].sum(1)[:, None, None, None]
        P = W if m is None else torch.einsum("li,bljk->bijk", m, W)
        val = ((P * Z / D).sum((1, 2, 3)) * wt).sum()
        total += val.detach()
        if cot is None:
            continue
        (cot * val).backward()
        dG = G.grad.view(6 * nj, o, o * o)
        dA = torch.empty_like(A)
        dA[:, :, :o] = voo.grad
        at = 0
        for zz, cnt in zip(zvals, counts):
            i = order[at:at + cnt]
            dGz = dG[i].reshape(cnt * o, o * o)
            dA[i, :, o:] = (dGz @ t2z[zz].t()).view(cnt, o, v)
            grad["t2T"].view(v, v, o * o)[zz] += A[i, :, o:].reshape(cnt * o, v).t() @ dGz
            at += cnt
        grad["vvop"].view(v * v, o, n).index_add_(0, x * v + y, dA)
        dGo = dG.view(6 * nj, o * o, o)
        grad["vooo"].view(v, o * o, o).index_add_(0, x, -(dGo @ Tzy.transpose(1, 2)))
        t2b = grad["t2T"].view(v * v, o, o)
        t2b.index_add_(0, z * v + y, -(Ox.transpose(1, 2) @ dGo))
        t2b.index_add_(0, y * v + x, tyx.grad)
        grad["t1T"].index_add_(0, z, t1z.grad)
        grad["fvo"].index_add_(0, z, fz.grad)
        grad["mo_energy"] += e.grad
        if mat_bar is not None:
            mat_bar += m.grad
        del G, A, dA, dG, dGo, V, W, Y, Z, P, D, val, voo, tyx, Ox, Tzy
    return total, grad, mat_bar


def _sorted_weights(abc):
    """Twice the symmetry factor of each sorted triple."""
    a, b, c = np.asarray(abc).T
    return 2.0 * np.where(a == c, 1 / 6, np.where((a == b) | (b == c), 0.5, 1.0))


def _all_sorted(v):
    t = np.stack(np.meshgrid(*[np.arange(v)] * 3, indexing="ij"), -1).reshape(-1, 3)
    return t[(t[:, 0] >= t[:, 1]) & (t[:, 1] >= t[:, 2])]


def _tril_pos(v):
    """(v, v) positions of the elements of a symmetric matrix in its packed lower triangle."""
    i, j = (torch.as_tensor(q, device="cuda") for q in np.tril_indices(v))
    pos = torch.zeros((v, v), dtype=torch.int64, device="cuda")
    pos[i, j] = torch.arange(len(i), device="cuda")
    pos[j, i] = pos[i, j]
    return pos.reshape(-1)


def _unpack(p, v):
    return p[..., _tril_pos(v)].view(*p.shape[:-1], v, v)


def _to_layouts(x, o, v):
    ovvv = _unpack(x["ovvv"], v)
    vvop = torch.cat([x["ovov"].permute(1, 3, 0, 2), ovvv.permute(1, 3, 0, 2)], dim=3)
    return dict(mo_energy=x["mo_energy"] * 1.0, t1T=x["t1"].t().contiguous(),
                t2T=x["t2"].permute(2, 3, 1, 0).contiguous(), vooo=x["ovoo"].permute(1, 0, 3, 2).contiguous(),
                fvo=x["fock"][o:, :o].contiguous(), vvop=vvop.contiguous())


def _iter64(s, o, v):
    """The 6-D solver with plain einsums, arrays as [i,j,k,a,b,c]."""
    full = _unpack(s["ovvv"], v)
    fock = s["fock"]
    t2T = s["t2"].permute(2, 3, 0, 1)
    w = torch.einsum("iabf,kjcf->ijkabc", full, s["t2"])
    w -= torch.einsum("iamj,mkbc->ijkabc", s["ovoo"], s["t2"])
    vt = 0.5 * (torch.einsum("iajb,kc->ijkabc", s["ovov"], s["t1"])
                + torch.einsum("abij,ck->ijkabc", t2T, fock[o:, :o]))

    def sym(x, perms):
        return sum(x.permute(*p, *[3 + i for i in p]) for p in perms)

    P6, P3 = R6, ((0, 1, 2), (1, 0, 2), (2, 1, 0))
    mo = s["mo_energy"]
    d = mo[:o, None] - mo[None, o:]
    d3 = d[:, None, None, :, None, None] + d[None, :, None, None, :, None] + d[None, None, :, None, None, :]
    W = sym(w, P6)
    wgt = (4 * W + W.permute(2, 0, 1, 3, 4, 5) + W.permute(1, 2, 0, 3, 4, 5) - 2 * W.permute(2, 1, 0, 3, 4, 5)
           - 2 * W.permute(0, 2, 1, 3, 4, 5) - 2 * W.permute(1, 0, 2, 3, 4, 5)) / 3
    seed = sym(w + vt, P6) / d3
    del w, vt, W
    foo, fvv = fock[:o, :o].clone(), fock[o:, o:].clone()
    foo.diagonal().zero_()
    fvv.diagonal().zero_()
    t3, e, conv = seed, float((seed * wgt).sum()), False
    for _ in range(50):
        u = torch.einsum("ae,ijkebc->ijkabc", fvv, t3) - torch.einsum("im,mjkabc->ijkabc", foo, t3)
        new = seed + sym(u, P3) / d3
        norm = float((new - t3).norm())
        t3, last = new, e
        e = float((t3 * wgt).sum())
        if abs(e - last) < 1e-8 and norm < 1e-6:
            conv = True
            break
    return conv, e, t3


def exact(case, seed):
    o, v, call = case["o"], case["v"], case["call"]
    s = prepare(case, seed)
    if call == "energy":
        abc = _all_sorted(v)
        return _triples64(s["L"], abc, _sorted_weights(abc))[0]
    if call in ("vjp", "block"):
        abc = _all_sorted(v) if call == "vjp" else np.asarray(_block_abc(v, case["slab"]))
        e, g, _ = _triples64(s["L"], abc, _sorted_weights(abc), cot=1.0)
        return e, g
    if call == "lno":
        t = np.stack(np.meshgrid(*[np.arange(v)] * 3, indexing="ij"), -1).reshape(-1, 3)
        t = t[t[:, 1] >= t[:, 2]]
        if len(t) * 36.0 * o ** 3 * (o + v) > 3e14:
            return None
        e, g, mb = _triples64(s["L"], t, np.where(t[:, 1] == t[:, 2], 0.5, 1.0), cot=2.0 / 3.0, mat=s["mat"])
        return e, mb, g
    if call == "df":
        naux = s["Lov"].shape[0]
        fac = [s[k].detach().clone().requires_grad_() for k in ("Loo", "Lov", "Lvv")]
        Lov = fac[1].view(naux, o, v)
        R = torch.cat([Lov, _unpack(fac[2], v)], dim=1)
        vvop = torch.einsum("Pia,Ppy->ayip", Lov, R)
        vooo = torch.einsum("Pia,Pjk->aikj", Lov, fac[0].view(naux, o, o))
        bars = torch.autograd.grad((vvop, vooo), fac, (s["bars"]["vvop"], s["bars"]["vooo"]))
        return dict(vvop=vvop.detach(), vooo=vooo.detach(), t2T=s["t2"].permute(2, 3, 1, 0).contiguous(), bars=bars)
    if call == "iter":
        conv, e, t3 = _iter64(s, o, v)
        return None, e, t3
    x = {k: s[k].detach().clone().requires_grad_() for k in ("t1", "t2", "mo_energy", "fock", "ovoo", "ovov", "ovvv")}
    L = _to_layouts(x, o, v)
    abc = _all_sorted(v)
    e, g, _ = _triples64({k: q.detach() for k, q in L.items()}, abc, _sorted_weights(abc), cot=1.0)
    return e, torch.autograd.grad([L[k] for k in KEYS], [x[k] for k in ("t1", "t2", "mo_energy", "fock", "ovoo",
                                                                        "ovov", "ovvv")], [g[k] for k in KEYS])
