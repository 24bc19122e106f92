"""Work that programs on this library have it do, as timed cases.

Six kinds of pass, each through the entry points that a program calls:

  t3_step   the T3 half of one RCCSDT iteration on resident amplitudes (dcc.t3_iteration):
            T3 -> r1, r2, W_vooo, W_vvvo, the T3 residual, symmetrize, divide, t3 += r3
  t3_vjp    the T3 residual and its vector-Jacobian product (dcc.adjoint), forward + backward
  q_energy  the (Q) energies of a list of virtual-block groups with a planned handle (dcc.rccsdt_q)
  t4_step   one T4 update of RCCSDTQ (dcc.graph.T4Iteration): residual, projector, divide, t4 += r4
  t3_blocks the batched T3 block helpers on canonical blocks (dcc._c_rccsdt): transpose-add, the
            three spin-summed variants, P3_full out of place
  diis      a new DIIS history over a T3-sized vector: the first record and one full subspace

The inputs have the shapes, symmetries and value distributions of dcc.synthetic (orbital
energies, 8-fold symmetric ERIs of 0.1, t2 of 1e-2, t3 of 1e-3, t4 of 1e-4), made here with torch
alone so that exact() can use the same ones.  exact() evaluates the textbook form of each pass
in FP64: full ordered tensors, every string once, permutation sums last.
"""
from __future__ import annotations

import itertools
import math
import os
import sys
import types

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "distributed-cc_b200"))

f64 = torch.float64
DEV = "cuda"


def _t3(name, nocc, nvir, precision):
    return {"name": name, "kind": "t3_step", "nocc": nocc, "nvir": nvir, "precision": precision}


def listed():
    return [
        # a production-size iteration (the secondary benchmark shape): tensor-core GEMMs and
        # gigabyte passes over T3
        _t3("t3_step_o10_v90", 10, 90, "bf16x3"),
        # odd virtual count (rows not a multiple of 16 bytes), the virtual space of the benchmark
        _t3("t3_step_o8_v93", 8, 93, "bf16x3"),
        # a medium molecule, where no pass fills the chip for long
        _t3("t3_step_o6_v40", 6, 40, "bf16x3"),
        # a test-size molecule: launches and host calls
        _t3("t3_step_o4_v9", 4, 9, "bf16x3"),
        # the plain FP64 path that the split precisions are checked against
        _t3("t3_step_o6_v40_fp64", 6, 40, "fp64"),
        # derivative of the residual (Lambda equations): forward and backward
        {"name": "t3_vjp_o6_v40", "kind": "t3_vjp", "nocc": 6, "nvir": 40, "precision": "bf16x3"},
        # a sample of the (Q) groups of a production-size molecule
        {"name": "q_o10_v90", "kind": "q_energy", "nocc": 10, "nvir": 90, "blksize": 4, "groups": 5,
         "precision": "bf16x3"},
        # every (Q) group of a small molecule
        {"name": "q_o5_v14", "kind": "q_energy", "nocc": 5, "nvir": 14, "blksize": 4, "groups": 0,
         "precision": "bf16x3"},
        # a T4 update at the N2 6-31G shape
        {"name": "t4_step_o7_v11", "kind": "t4_step", "nocc": 7, "nvir": 11, "precision": "bf16x3"},
        # a small T4 update in plain FP64
        {"name": "t4_step_o5_v8_fp64", "kind": "t4_step", "nocc": 5, "nvir": 8, "precision": "fp64"},
        # the block helpers as a drop-in caller uses them, on every canonical block
        {"name": "t3_blocks_o8_v90", "kind": "t3_blocks", "nocc": 8, "nvir": 90},
        # the extrapolation of a medium T3 vector, six slots
        {"name": "diis_o8_v60", "kind": "diis", "nocc": 8, "nvir": 60, "space": 6},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    while True:
        kind = rng.choice(["t3_step", "t3_step", "t3_step", "t3_vjp", "q_energy", "t4_step", "t4_step", "t3_blocks",
                           "diis"])
        prec = rng.choice(["bf16x3", "bf16x3", "bf16x3", "tf32x3", "fp64"])
        if kind == "t3_step":
            c = {"kind": kind, "nocc": rng.randint(3, 10), "nvir": _log_int(rng, 7, 104), "precision": prec}
            lim = 1.3e12 if prec == "fp64" else 2.6e12 if prec == "tf32x3" else 1.2e13
        elif kind == "t3_vjp":
            c = {"kind": kind, "nocc": rng.randint(3, 6), "nvir": _log_int(rng, 7, 44), "precision": prec}
            lim = 6e11
        elif kind == "q_energy":
            c = {"kind": kind, "nocc": rng.randint(3, 10), "nvir": _log_int(rng, 8, 93), "blksize": rng.choice([3, 4]),
                 "groups": rng.randint(2, 5), "precision": rng.choice(["bf16x3", "bf16x3", "tf32x3", "fp64"])}
            lim = 4e11 if c["precision"] == "bf16x3" else 1.5e11
        elif kind == "t4_step":
            c = {"kind": kind, "nocc": rng.randint(3, 7), "nvir": rng.randint(4, 12), "precision": prec}
            lim = 1.2 * work({"kind": kind, "nocc": 7, "nvir": 11, "precision": prec})["flops"]
        elif kind == "t3_blocks":
            c = {"kind": kind, "nocc": rng.randint(2, 10), "nvir": _log_int(rng, 7, 112)}
            lim = None
        else:
            c = {"kind": kind, "nocc": rng.randint(2, 10), "nvir": _log_int(rng, 7, 90), "space": rng.randint(3, 8)}
            lim = None
        n = c["nocc"] * (c["nocc"] + 1) * (c["nocc"] + 2) // 6 * c["nvir"] ** 3
        if lim is None:
            if n <= 120 * 90 ** 3 and n * c.get("space", 1) <= 160 * 10 ** 6:
                return c
        elif work(c)["flops"] <= lim and c["nocc"] ** 3 * c["nvir"] ** 3 <= 10 ** 3 * 90 ** 3:
            return c


# ---------------------------------------------------------------- inputs

def _canonical(no):
    return [(i, j, k) for i in range(no) for j in range(i, no) for k in range(j, no)]


def _stored4(no):
    """T4 blocks that are kept: i<=j<=k<=l without three equal indices."""
    return [(i, j, k, l) for i in range(no) for j in range(i, no) for k in range(j, no) for l in range(k, no)
            if not (i == j == k or j == k == l)]


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _randn(g, *shape, scale=1.0):
    return torch.randn(*shape, dtype=f64, device=DEV, generator=g).mul_(scale)


def _sym_blocks(x, no, nv, rows, n):
    """Rows of x [no^n, nv^n axes] summed over the simultaneous permutations, / n!: the blocks
    of a tensor invariant under them."""
    x = x.view((no,) * n + (nv,) * n)
    idx = torch.tensor(rows, device=DEV)
    out = torch.zeros((len(rows),) + (nv,) * n, dtype=f64, device=DEV)
    for p in itertools.permutations(range(n)):
        inv = [p.index(m) for m in range(n)]
        out += x[tuple(idx[:, m] for m in p)].permute(0, *(1 + m for m in inv))
    return out.div_(math.factorial(n))


def _physicist(g, no, nv):
    """<pq|rs> with the 8-fold symmetry of real integrals, and e_occ, e_vir."""
    n = no + nv
    x = _randn(g, n, n, n, n, scale=0.1)
    x = x + x.transpose(0, 1)
    x = x + x.transpose(2, 3)
    x = (x + x.permute(2, 3, 0, 1)).div_(8.0)
    eo = (torch.rand(no, dtype=f64, device=DEV, generator=g) * 1.2 - 1.5).sort().values
    ev = (torch.rand(nv, dtype=f64, device=DEV, generator=g) * 2.9 + 0.1).sort().values
    return x.permute(0, 2, 1, 3), eo, ev


def _inputs(case, seed):
    """The integral slices, amplitudes and energies of the coupled-cluster kinds."""
    g, no, nv = _gen(seed), case["nocc"], case["nvir"]
    phys, eo, ev = _physicist(g, no, nv)
    o, v = slice(0, no), slice(no, None)
    d = types.SimpleNamespace(no=no, nv=nv, e_occ=eo, e_vir=ev, eia=(eo[:, None] - ev[None, :]).contiguous())
    cut = lambda *s: phys[s].contiguous()  # noqa: E731
    d.W_vvvv, d.W_vvvo, d.W_vooo = cut(v, v, v, v), cut(v, v, v, o), cut(v, o, o, o)
    d.W_ovov, d.W_ovvo, d.W_oooo = cut(o, v, o, v), cut(o, v, v, o), cut(o, o, o, o)
    d.vvoo, d.oovv, d.vovv, d.ooov = cut(v, v, o, o), cut(o, o, v, v), cut(v, o, v, v), cut(o, o, o, v)
    if case["kind"] == "t4_step":
        d.eris = phys.contiguous()
    t2 = _randn(g, no, no, nv, nv, scale=1e-2)
    d.t2 = (0.5 * (t2 + t2.permute(1, 0, 3, 2))).contiguous()
    cv, co = _randn(g, nv, nv, scale=1e-2), _randn(g, no, no, scale=1e-2)
    d.F_vv = (torch.diag(ev) + 0.5 * (cv + cv.t())).contiguous()
    d.F_oo = (torch.diag(eo) + 0.5 * (co + co.t())).contiguous()
    d.fock_ov = _randn(g, no, nv, scale=1e-2)
    d.ijk = torch.tensor(_canonical(no), dtype=torch.int32, device=DEV)
    if case["kind"] == "t4_step":
        every3 = list(itertools.product(range(no), repeat=3))
        d.t3 = _sym_blocks(_randn(g, no ** 3, nv ** 3, scale=1e-3), no, nv, every3, 3).view((no,) * 3 + (nv,) * 3)
        d.t4 = _sym_blocks(_randn(g, no ** 4, nv ** 4, scale=1e-4), no, nv, _stored4(no), 4)
        d.ijkl = torch.tensor(_stored4(no), dtype=torch.int32, device=DEV)
    else:
        d.t3 = _sym_blocks(_randn(g, no ** 3, nv ** 3, scale=1e-3), no, nv, _canonical(no), 3)
    return d


def _q_groups(case):
    """The case's (a0, a1, b0, b1, c0, c1) groups: all of them, or some spread over the list."""
    nv, blk = case["nvir"], case["blksize"]
    ranges = [(x, min(x + blk, nv)) for x in range(0, nv, blk)]
    g = [a + b + c for n, c in enumerate(ranges) for m, b in enumerate(ranges[:n + 1]) for a in ranges[:m + 1]]
    k = case["groups"]
    if not k or k >= len(g):
        return g
    return [g[(2 * n + 1) * len(g) // (2 * k)] for n in range(k)]


def _diis_vectors(case, seed):
    """Iterates that converge towards a fixed vector, as amplitudes do: [lower | t3] per iteration."""
    g, no, nv = _gen(seed), case["nocc"], case["nvir"]
    n3 = len(_canonical(no)) * nv ** 3
    n12 = no * nv + no * (no + 1) // 2 * nv * nv
    fixed = [_randn(g, n12, scale=1e-2), _randn(g, n3, scale=1e-3)]
    return [[(x + _randn(g, x.numel(), scale=s * 0.6 ** (k + 1))) for x, s in zip(fixed, (1e-2, 1e-3))]
            for k in range(case["space"] + 1)]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "diis":
        from dcc.diis import DIIS
        vec = _diis_vectors(case, seed)
        return {"kind": kind, "vec": vec, "work": [torch.empty_like(x) for x in vec[0]], "diis": DIIS(case["space"], DEV)}
    if kind == "t3_blocks":
        n = len(_canonical(case["nocc"]))
        A = _randn(_gen(seed), n, case["nvir"], case["nvir"], case["nvir"], scale=1e-3)
        return {"kind": kind, "A": A, "nvir": case["nvir"], "out": [torch.empty_like(A) for _ in range(5)]}
    d = _inputs(case, seed)
    no, nv = d.no, d.nv
    if kind == "t3_step":
        from dcc.t3_iteration import T3Iteration
        return {"kind": kind, "d": d, "it": T3Iteration(no, nv, case["precision"]), "t3": torch.empty_like(d.t3)}
    if kind == "t3_vjp":
        args = [getattr(d, n).requires_grad_() for n in _VJP_ARGS]
        return {"kind": kind, "args": args, "lam": _randn(_gen(seed + 7919), *d.t3.shape), "precision": case["precision"]}
    if kind == "q_energy":
        from dcc import _c_rccsdt, rccsdt_q
        er = {"vvvo": d.W_vvvo, "vooo": d.W_vooo, "vvoo": d.vvoo, "ovvo": d.W_ovvo, "ovov": d.W_ovov, "vvvv": d.W_vvvv,
              "oooo": d.W_oooo}
        groups = _q_groups(case)
        q = rccsdt_q.QEnergy(no, nv, case["blksize"], case["precision"])
        q.prepare(groups)
        return {"kind": kind, "q": q, "er": er, "t2": d.t2.permute(2, 3, 0, 1).contiguous(), "groups": groups,
                "t3_abc": _c_rccsdt.redistribute_ijk_to_abc(d.t3, no, nv), "e_occ": d.e_occ, "e_vir": d.e_vir}
    from dcc.graph import T4Iteration
    start = d.t4.clone()
    return {"kind": kind, "start": start, "it": T4Iteration(d, case["precision"])}


_VJP_ARGS = ("t2", "t3", "F_vv", "F_oo", "W_vvvo", "W_vooo", "W_vvvv", "W_ovov", "W_ovvo", "W_oooo")


def run(s):
    kind = s["kind"]
    if kind == "t3_step":
        it, d, t3 = s["it"], s["d"], s["t3"]
        t3.copy_(d.t3)
        dr1, dr2 = it.feedback_r1r2(t3, d.fock_ov, d.oovv, d.vovv, d.ooov)
        x = types.SimpleNamespace(**vars(d))
        x.W_vooo, x.W_vvvo = d.W_vooo.clone(), d.W_vvvo.clone()  # rebuilt by the caller every iteration
        it.feedback_w(x.W_vooo, x.W_vvvo, d.oovv)
        it.residual(x, t3)
        norms = it.update(t3, d.eia)
        return {"dr1": dr1, "dr2": dr2, "W_vooo": x.W_vooo, "W_vvvo": x.W_vvvo, "t3": t3, "norms": norms}
    if kind == "t3_vjp":
        from dcc import adjoint
        r3 = adjoint.t3_residual_fn(*s["args"], precision=s["precision"])
        return [r3.detach()] + list(torch.autograd.grad(r3, s["args"], s["lam"]))
    if kind == "q_energy":
        q = s["q"]
        q.out.zero_()
        return q.run(s["er"], s["t2"], s["t3_abc"], s["e_occ"], s["e_vir"], s["groups"])
    if kind == "t4_step":
        it = s["it"]
        it.d.t4.copy_(s["start"])
        norms = it.step()
        return {"t4": it.d.t4, "norms": norms}
    if kind == "t3_blocks":
        from dcc import _c_rccsdt as c
        A, nv, (T, B0, B1, B2, P) = s["A"], s["nvir"], s["out"]
        c.t3_transpose_add_(A, T, nv)
        c.t3_spin_summation_triple_sym_(A, B0, B1, B2, nv)
        c.t3_spin_summation(A, P, A.shape[0], nv, "P3_full", -1.0 / 6.0, 1.0)
        return s["out"]
    s["diis"].reset()
    norms = []
    for v in s["vec"]:
        for w, x in zip(s["work"], v):
            w.copy_(x)
        s["diis"].update(s["work"])
        norms.append(s["diis"].last_delta_norm_sq)
    return {"lower": s["work"][0], "t3": s["work"][1], "norm": norms[-1]}


# ---------------------------------------------------------------- work and tolerance

def work(case):
    no, nv, kind = case["nocc"], case["nvir"], case["kind"]
    n3, n = no * (no + 1) * (no + 2) // 6, no + nv
    tri, t3 = n3 * nv ** 3, no ** 3 * nv ** 3
    ints = nv ** 4 + no * nv ** 3 + 3 * no ** 2 * nv ** 2 + no ** 3 * nv + no ** 4
    if kind in ("t3_step", "t3_vjp"):
        # W_vvvv.t3 and F_vv.t3 on canonical blocks; W.t2, W_ovov / W_ovvo and W_oooo / F_oo on
        # ordered ones
        r3 = 6.0 * tri * (nv ** 2 + nv) + 2.0 * t3 * (nv + no + 3 * no * nv + no ** 2 + no)
        if kind == "t3_vjp":
            return {"flops": 3 * r3, "bytes": 8.0 * (4 * tri + 2 * ints)}
        fb = 2.0 * t3 * (2 * nv + 2 * no + 1)
        return {"flops": r3 + fb, "bytes": 8.0 * (2 * tri + ints + 3 * no * nv ** 3 + 2 * no ** 2 * nv ** 2)}
    if kind == "q_energy":
        el = t2 = 0.0
        for a0, a1, b0, b1, c0, c1 in _q_groups(case):
            el += (a1 - a0) * (b1 - b0) * (c1 - c0) * (nv - c0) * no ** 4
            t2 += ((a1 - a0) * (b1 - b0) * (c1 - c0) * nv * no ** 2
                   + (nv - c0) * nv * no ** 2 * ((a1 - a0) * (b1 - b0) + (a1 - a0) * (c1 - c0) + (b1 - b0) * (c1 - c0)))
        # 12 strings each over vvvo, vooo, W_vvvvoo, W_vvoooo; the builds of W_vvvvoo (six strings)
        return {"flops": el * 2.0 * 24 * (nv + no) + t2 * 3.0 * 4.0 * (nv + 2 * no),
                "bytes": 8.0 * (nv * (nv + 1) * (nv + 2) // 6 * no ** 3 + ints)}
    if kind == "t4_step":
        n4, t4 = len(_stored4(no)), nv ** 4
        per = 12 * (2 * nv + 2 * no + no + no ** 2) + 36 * no * nv + 6 * nv ** 2 + 4 * nv + 4 * no + 6 * no ** 2 + 20 * no * nv
        build = no ** 3 * nv ** 3 * (4 * no * nv + no * nv) + 2 * no ** 4 * nv ** 4 * nv * no
        return {"flops": 2.0 * (n4 * t4 * per + build), "bytes": 8.0 * (2 * n4 * t4 + no ** 3 * nv ** 3 + n ** 4 + ints)}
    if kind == "t3_blocks":
        return {"flops": 13.0 * tri, "bytes": 8.0 * 6 * tri}
    vec = tri + no * nv + no * (no + 1) // 2 * nv ** 2
    # per iteration: the iterate in and out, the slots' error vectors for the inner products and
    # the slots for the combination
    k = case["space"]
    return {"flops": 4.0 * vec * k * (k + 1) / 2, "bytes": 8.0 * vec * (4 * k + k * (k + 1))}


# about four times the largest deviation from exact() over the listed sizes and some fifty draws
# (t3_step 3.0e-5 in r2's T3 part, whose contraction runs over nocc nvir^2 terms; t3_vjp 5.1e-5;
# q_energy 6.0e-7; t4_step 1.2e-6; FP64 2.3e-15, where another order of the sums is allowed for)
_REL = {
    ("t3_step", "fp64"): 2e-14, ("t3_step", "bf16x3"): 1.2e-4, ("t3_step", "tf32x3"): 1.2e-4,
    ("t3_vjp", "fp64"): 2e-14, ("t3_vjp", "bf16x3"): 1.4e-4, ("t3_vjp", "tf32x3"): 2e-4,
    ("q_energy", "fp64"): 1e-11, ("q_energy", "bf16x3"): 2.5e-6, ("q_energy", "tf32x3"): 2.5e-6,
    ("t4_step", "fp64"): 2e-14, ("t4_step", "bf16x3"): 5e-6, ("t4_step", "tf32x3"): 5e-6,
}


def tolerance(case):
    if case["kind"] == "t3_blocks":
        return {"rel": 5e-16}
    if case["kind"] == "diis":
        return {"rel": 2e-13}
    return {"rel": _REL[case["kind"], case["precision"]]}


# ---------------------------------------------------------------- FP64 answers

def _unpack3(t3, no):
    """Every ordered (x,y,z) of canonical blocks."""
    index = {q: n for n, q in enumerate(_canonical(no))}
    rows = {}
    for f, o in enumerate(itertools.product(range(no), repeat=3)):
        order = sorted(range(3), key=lambda p: (o[p], p))
        rank = tuple(order.index(p) for p in range(3))
        rows.setdefault(rank, ([], []))
        rows[rank][0].append(f)
        rows[rank][1].append(index[tuple(o[p] for p in order)])
    out = torch.empty((no ** 3,) + tuple(t3.shape[1:]), dtype=f64, device=DEV)
    for rank, (dst, src) in rows.items():
        out = out.index_copy(0, torch.tensor(dst, device=DEV),
                             t3[torch.tensor(src, device=DEV)].permute(0, *(1 + r for r in rank)))
    return out.view((no,) * 3 + tuple(t3.shape[1:]))


def _r3(d, t3, U):
    """compute_r3_tri on canonical blocks: the ordered strings, their sum over the simultaneous
    permutations, and W_vvvv.t3 + F_vv.t3."""
    no, nv, e = d.no, d.nv, torch.einsum
    G = -0.5 * (d.W_ovov + d.W_ovvo.permute(0, 1, 3, 2))
    parts = []
    for j in range(no):
        s = e('abd,ikdc->ikabc', d.W_vvvo[..., j], d.t2) - e('ali,lkbc->ikabc', d.W_vooo[..., j], d.t2)
        s = s - e('lbid,kldca->ikabc', d.W_ovov, U[j]) + e('laid,kldcb->ikabc', G, U[j])
        s = s + 0.5 * e('ladi,klbcd->ikabc', d.W_ovvo, U[j])
        s = s + 0.5 * e('lmi,lmkabc->ikabc', d.W_oooo[..., j], U) - 0.5 * e('li,lkabc->ikabc', d.F_oo, U[:, j])
        parts.append(s)
    S = torch.stack(parts, 1)
    del parts
    ijk = torch.tensor(_canonical(no), device=DEV)
    r = (e('abde,qdec->qabc', d.W_vvvv, t3) + e('acde,qdbe->qabc', d.W_vvvv, t3) + e('bcde,qade->qabc', d.W_vvvv, t3)
         + e('ad,qdbc->qabc', d.F_vv, t3) + e('bd,qadc->qabc', d.F_vv, t3) + e('cd,qabd->qabc', d.F_vv, t3))
    for p in itertools.permutations(range(3)):
        inv = [p.index(m) for m in range(3)]
        r = r + S[tuple(ijk[:, m] for m in p)].permute(0, *(1 + m for m in inv))
    return r


def _exact_t3_step(d):
    no, nv, e = d.no, d.nv, torch.einsum
    U = _unpack3(d.t3, no)
    X = 2.0 * U - U.permute(0, 1, 2, 5, 4, 3) - U.permute(0, 1, 2, 4, 3, 5)
    dr2 = 0.5 * e('xa,xyzabc->yzbc', d.fock_ov, X) + e('cxad,xyzdba->yzbc', d.vovv, X) - e('zxla,xyzabc->ylbc', d.ooov, X)
    W_vooo = d.W_vooo + e('mxde,xyzead->amyz', d.oovv, X)
    W_vvvo = d.W_vvvo - e('zxde,xyzeba->abdy', d.oovv, X)
    del X
    t = d.t3
    c = 2.0 * t - t.permute(0, 3, 2, 1) - t.permute(0, 2, 1, 3)
    V = 2.0 * c - c.permute(0, 1, 3, 2)
    del c
    dr1 = torch.zeros(no, nv, dtype=f64, device=DEV)
    for q, (i, j, k) in enumerate(_canonical(no)):
        if i == j == k:
            continue
        c1, c2, c3 = (1.0, 1.0, 1.0) if i < j < k else (1.0, 0.0, 0.5) if i == j else (0.5, 1.0, 0.0)
        dr1[i] += c1 * e('bc,abc->a', d.oovv[j, k], V[q])
        dr1[j] += c2 * e('bc,bac->a', d.oovv[i, k], V[q])
        dr1[k] += c3 * e('bc,bca->a', d.oovv[i, j], V[q])
    del V
    x = types.SimpleNamespace(**vars(d))
    x.W_vooo, x.W_vvvo = W_vooo, W_vvvo
    r = _r3(x, t, U)
    del U
    s = sum(r.permute(0, *(1 + m for m in p)) for p in itertools.permutations(range(3)))
    r = r - s / 6.0
    ijk = d.ijk.long()
    r = r / (d.eia[ijk[:, 0]][:, :, None, None] + d.eia[ijk[:, 1]][:, None, :, None] + d.eia[ijk[:, 2]][:, None, None, :])
    return {"dr1": dr1, "dr2": dr2, "W_vooo": W_vooo, "W_vvvo": W_vvvo, "t3": t + r,
            "norms": r.square().sum().expand(2).clone()}


def _exact_vjp(d, lam):
    x = types.SimpleNamespace(no=d.no, nv=d.nv)
    args = [getattr(d, n).clone().requires_grad_() for n in _VJP_ARGS]
    for n, a in zip(_VJP_ARGS, args):
        setattr(x, n, a)
    x.W_oooo = 0.5 * (x.W_oooo + x.W_oooo.permute(1, 0, 3, 2))
    r = _r3(x, x.t3, _unpack3(x.t3, d.no))
    g = list(torch.autograd.grad(r, args, lam))
    # t3 lives on blocks symmetric under the permutations that leave (i,j,k) alone
    for q, (i, j, k) in enumerate(_canonical(d.no)):
        o = (i, j, k)
        stab = [p for p in itertools.permutations(range(3)) if tuple(o[m] for m in p) == o]
        if len(stab) > 1:
            g[1][q] = sum(g[1][q].permute(p) for p in stab) / len(stab)
    return [r.detach()] + g


def _swap(x, i, j):
    return x.transpose(i, j)


def _exact_q(case, d):
    """[Q] and (Q): connected T3 and T2 quadruples of every group as sums over the permutations of
    four (virtual range, occupied index) pairs."""
    no, nv, e = d.no, d.nv, torch.einsum
    t2 = d.t2.permute(2, 3, 0, 1)
    T = _unpack3(d.t3, no).permute(3, 4, 5, 0, 1, 2)
    eb = ep = 0.0
    for a0, a1, b0, b1, c0, c1 in _q_groups(case):
        R = [slice(a0, a1), slice(b0, b1), slice(c0, c1), slice(c0, nv)]
        n = [r.stop - r.start for r in R]
        z = torch.zeros(tuple(n) + (no,) * 4, dtype=f64, device=DEV)
        x, sq = torch.zeros_like(z), torch.zeros_like(z)
        for p in itertools.permutations(range(4)):
            A, B, C, D = (R[m] for m in p)
            W = (0.5 * e('abef,fcjk->abcejk', d.W_vvvv[A, B], t2[:, C]) + 0.5 * e('acef,fbkj->abcejk', d.W_vvvv[A, C], t2[:, B])
                 - e('mbej,acmk->abcejk', d.W_ovvo[:, B], t2[A, C]) - e('mcek,abmj->abcejk', d.W_ovvo[:, C], t2[A, B])
                 - e('maje,bcmk->abcejk', d.W_ovov[:, A], t2[B, C]) - e('make,cbmj->abcejk', d.W_ovov[:, A], t2[C, B]))
            Y = -0.5 * e('mnki,abnj->abmijk', d.W_oooo, t2[A, B]) - 0.5 * e('mnkj,bani->abmijk', d.W_oooo, t2[B, A])
            base = e('cdel,abeijk->abcdijkl', d.W_vvvo[C, D], T[A, B]) - e('dmli,abcmjk->abcdijkl', d.W_vooo[D], T[A, B][:, :, C])
            back = [p.index(m) for m in range(4)]
            back = back + [4 + m for m in back]
            z += 0.5 * base.permute(back)
            base = e('abcejk,edil->abcdijkl', W, t2[:, D]) - e('abmijk,cdml->abcdijkl', Y, t2[C, D])
            x += 0.5 * base.permute(back)
            sq += 0.25 * e('abij,cdkl->abcdijkl', d.vvoo[A, B], t2[C, D]).permute(back)
        E = lambda r, ax: d.e_vir[r].view([-1 if m == ax else 1 for m in range(8)])  # noqa: E731
        O = lambda ax: d.e_occ.view([-1 if m == ax else 1 for m in range(8)])  # noqa: E731
        x = (x + z) / (O(4) + O(5) + O(6) + O(7) - E(R[0], 0) - E(R[1], 1) - E(R[2], 2) - E(R[3], 3))
        x = 2.0 * x - _swap(x, 4, 5) - _swap(x, 4, 6) - _swap(x, 4, 7)
        x = 2.0 * x - _swap(x, 5, 6) - _swap(x, 5, 7)
        x = 2.0 * x - _swap(x, 6, 7)
        i = [torch.arange(r.start, r.stop, device=DEV).view([-1 if m == ax else 1 for m in range(4)]) for ax, r in enumerate(R)]
        ok = (i[0] <= i[1]) & (i[1] <= i[2]) & (i[2] <= i[3]) & ~((i[0] == i[1]) & (i[1] == i[2]))
        ok = ok & ~((i[1] == i[2]) & (i[2] == i[3]))
        eq = (i[0] == i[1]).to(f64) + (i[1] == i[2]).to(f64) + (i[2] == i[3]).to(f64)
        x *= (24.0 / 2.0 ** eq * ok.to(f64))[..., None, None, None, None]
        b = float((x * sq).sum()) / 12.0
        eb += b
        ep += float((x * z).sum()) / 12.0 + b
    return torch.tensor([eb, ep], dtype=f64)


def _unpack4(t4, no):
    nv = t4.shape[1]
    index = {q: n for n, q in enumerate(_stored4(no))}
    rows = {}
    for f, o in enumerate(itertools.product(range(no), repeat=4)):
        order = sorted(range(4), key=lambda p: (o[p], p))
        can = tuple(o[p] for p in order)
        if can in index:
            rank = tuple(order.index(p) for p in range(4))
            rows.setdefault(rank, ([], []))
            rows[rank][0].append(f)
            rows[rank][1].append(index[can])
    out = torch.zeros((no ** 4,) + (nv,) * 4, dtype=f64, device=DEV)
    for rank, (dst, src) in rows.items():
        out[torch.tensor(dst, device=DEV)] = t4[torch.tensor(src, device=DEV)].permute(0, *(1 + r for r in rank))
    return out.view((no,) * 4 + (nv,) * 4)


def _exact_t4_step(d):
    """One T4 update over the full ordered space: each string once, divided by the number of
    permutations that leave it alone, then the sum over the 24 simultaneous permutations."""
    no, nv, e = d.no, d.nv, torch.einsum
    o, v = slice(0, no), slice(no, None)
    t2, t3, er = d.t2, d.t3, d.eris
    T = _unpack4(d.t4, no)
    t3p = 2.0 * t3 - _swap(t3, 3, 5) - _swap(t3, 3, 4)
    oovv, ovvv, ooov, oovo = er[o, o, v, v], er[o, v, v, v], er[o, o, o, v], er[o, o, v, o]
    A = 2.0 * e('maef,jibf->ijeabm', ovvv, t2) - e('mafe,jibf->ijeabm', ovvv, t2)
    A = A - 2.0 * e('mnei,njab->ijeabm', oovo, t2) + e('nmei,njab->ijeabm', oovo, t2)
    A = A + 0.5 * e('nmfe,nijfab->ijeabm', oovv, t3p) - 0.25 * e('mnfe,nijfab->ijeabm', oovv, t3p)
    W_oovvvo = A + A.permute(1, 0, 2, 4, 3, 5)
    W_ovovvo = (e('mafe,jibf->iejabm', ovvv, t2) - e('mnie,njab->iejabm', ooov, t2)
                - 0.5 * e('nmef,injfab->iejabm', oovv, t3))
    A = e('mnek,ijae->kjinma', oovo, t2) + 0.5 * e('mnef,ijkaef->kjinma', oovv, t3)
    W_ooooov = A + A.permute(1, 0, 2, 4, 3, 5)
    Ts = 2.0 * T - _swap(T, 4, 5) - _swap(T, 4, 6) - _swap(T, 4, 7)
    A = 0.5 * e('mief,ijklfabe->jklmab', oovv, Ts) + e('amef,ijkebf->ijkmab', er[v, o, v, v], t3)
    Wv = -0.5 * e('jief,ijklfabc->klabce', oovv, Ts)
    c2 = 2.0 * t2 - _swap(t2, 2, 3)
    x = (er[o, v, v, o] + e('nmfe,nifa->maei', oovv, c2) - 0.5 * e('mnfe,nifa->maei', oovv, c2)
         - 0.5 * e('nmef,infa->maei', oovv, t2))
    A = A + e('maei,jkbe->ijkmab', x, t2) + e('make,jibe->ijkmab', d.W_ovov, t2) - 0.5 * e('mnki,njab->ijkmab', d.W_oooo, t2)
    W_oooovv = A + A.permute(1, 0, 2, 3, 5, 4)
    W_oovvvv = Wv + Wv.permute(1, 0, 2, 4, 3, 5) + 0.5 * e('abef,xyfc->xyabce', d.W_vvvv, t2) + 0.5 * e('acef,yxfb->xyabce', d.W_vvvv, t2)
    Wsym = W_ovovvo + W_ovovvo.permute(2, 1, 0, 4, 3, 5)
    t3s = t3 + t3.permute(0, 1, 2, 4, 5, 3)
    R = 0.5 * e('abej,iklecd->ijklabcd', d.W_vvvo, t3) - 0.5 * e('amij,mklbcd->ijklabcd', d.W_vooo, t3)
    R += 0.125 * e('ijeabm,mklecd->ijklabcd', W_oovvvo, t3p) - e('iejcbm,mklaed->ijklabcd', W_ovovvo, t3)
    R += -0.125 * e('iejabm,mklced->ijklabcd', Wsym, t3s) + 0.5 * e('kjinma,mnlbcd->ijklabcd', W_ooooov, t3)
    R += -0.5 * e('ijkmab,mlcd->ijklabcd', W_oooovv, t2) + 0.5 * e('jkabce,iled->ijklabcd', W_oovvvv, t2)
    R += e('ae,ijklebcd->ijklabcd', d.F_vv, T) / 6.0 + 0.25 * e('abef,ijklefcd->ijklabcd', d.W_vvvv, T)
    R += -e('mi,mjklabcd->ijklabcd', d.F_oo, T) / 6.0 + 0.25 * e('mnij,mnklabcd->ijklabcd', d.W_oooo, T)
    R += e('maei,mjklebcd->ijklabcd', d.W_ovvo, Ts) / 12.0 - 0.5 * e('mbie,mjklaecd->ijklabcd', d.W_ovov, T)
    sw = _swap(T, 4, 5) + _swap(T, 4, 6) + _swap(T, 4, 7)
    R -= e('maie,mjklebcd->ijklabcd', d.W_ovov, sw) / 12.0
    del sw, Ts, T
    q = d.ijkl.long()
    r = torch.zeros_like(d.t4)
    for p in itertools.permutations(range(4)):
        inv = [p.index(m) for m in range(4)]
        r += R[tuple(q[:, m] for m in p)].permute(0, *(1 + m for m in inv))
    del R
    om = lambda y: sum(_swap(y, i, j) for i, j in itertools.combinations(range(1, 5), 2))  # noqa: E731
    x1 = om(r) - 6.0 * r
    x2 = om(x1) - 2.0 * x1
    x3 = om(x2)
    r = (2.0 * om(x3) + 19.0 * x3 + 48.0 * x2) / 576.0
    r = r / (d.eia[q[:, 0]][:, :, None, None, None] + d.eia[q[:, 1]][:, None, :, None, None]
             + d.eia[q[:, 2]][:, None, None, :, None] + d.eia[q[:, 3]][:, None, None, None, :])
    return {"t4": d.t4 + r, "norms": r.square().sum().expand(2).clone()}


def _exact_diis(case, seed):
    space = case["space"]
    vec = [torch.cat(v) for v in _diis_vectors(case, seed)]
    prev, xs, es, H, norm = vec[0], [], [], np.zeros((space + 1, space + 1)), 0.0
    H[0, 1:] = H[1:, 0] = 1.0
    for n, x in enumerate(vec[1:]):
        xs.append(x)
        es.append(x - prev)
        for i, y in enumerate(es):
            H[n + 1, i + 1] = H[i + 1, n + 1] = float(torch.dot(es[n], y))
        g = np.zeros(n + 2)
        g[0] = 1.0
        c = np.linalg.solve(H[:n + 2, :n + 2], g)
        new = sum(float(a) * y for a, y in zip(c[1:], xs))
        norm = float((new - prev).square().sum())
        prev = new
    n12 = case["nocc"] * case["nvir"] + case["nocc"] * (case["nocc"] + 1) // 2 * case["nvir"] ** 2
    return {"lower": prev[:n12], "t3": prev[n12:], "norm": norm}


def exact(case, seed):
    kind = case["kind"]
    if kind == "diis":
        return _exact_diis(case, seed)
    if kind == "t3_blocks":
        n, nv = len(_canonical(case["nocc"])), case["nvir"]
        A = _randn(_gen(seed), n, nv, nv, nv, scale=1e-3)
        acb, cba, bac = A.permute(0, 1, 3, 2), A.permute(0, 3, 2, 1), A.permute(0, 2, 1, 3)
        full = sum(A.permute(0, *(1 + m for m in p)) for p in itertools.permutations(range(3)))
        return [A + A.permute(0, 2, 3, 1), 2.0 * A - acb - cba, 2.0 * A - bac - acb, 2.0 * A - cba - bac, A - full / 6.0]
    d = _inputs(case, seed)
    if kind == "t3_step":
        return _exact_t3_step(d)
    if kind == "t3_vjp":
        return _exact_vjp(d, _randn(_gen(seed + 7919), *d.t3.shape))
    if kind == "q_energy":
        return _exact_q(case, d)
    return _exact_t4_step(d)
