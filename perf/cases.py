"""What a program that uses this package has it do, as cases that can be timed.

Each case is one call, or one short run of calls, of the public API
(lfric_core_b200.lfx) on a seeded cubed-sphere problem C<n> x <nl>. The sizes
are those of the benchmark's configurations, of the tests, and odd ones between
them. ``prepare`` makes what the program holds before the call: operator,
preconditioner, solver, right-hand side. ``run`` is the call.
"""
import math
import random

import numpy as np
import torch

from lfric_core_b200 import lfx
from lfric_core_b200 import meshgen as mg
from lfric_core_b200 import workloads as wl

_context = None


def _ctx():
    """One context for the process, as a program has it."""
    global _context
    if _context is None:
        _context = lfx.Context(0)
    return _context


def listed():
    return [
        # the smallest solve (the size of the smoke check): latency and launches
        dict(name="cg-w0-c8x6", kind="solve", method="cg", n=8, nl=6, r_tol=1e-8),
        # mass-matrix solve, FP64 Jacobi CG: the first configuration of the benchmark
        dict(name="cg-w0-c24x20", kind="solve", method="cg", n=24, nl=20, r_tol=1e-8),
        # an odd panel (greedy colouring), ragged column height, non-symmetric
        # method with the column preconditioner twice an iteration
        dict(name="bicgstab-w2-c37x23", kind="solve", method="bicgstab", n=37, nl=23, r_tol=1e-9),
        # the headline system, plain FP64 GMRES(10)
        dict(name="gmres-w2-c96x30", kind="solve", method="gmres", n=96, nl=30, r_tol=1e-8),
        # the headline: FP32 GMRES(10) inside FP64 refinement
        dict(name="refined-w2-c96x30", kind="solve", method="refined", n=96, nl=30, r_tol=1e-8),
        # 64 right-hand sides on the tensor cores, CG on each
        dict(name="mrhs-tf32-c48x30", kind="mrhs", method="cg", mma="tf32", n=48, nl=30,
             r_tol=1e-10),
        # the same as one block, BF16 operands, on a smaller mesh
        dict(name="mrhs-block-bf16-c24x20", kind="mrhs", method="block", mma="bf16", n=24, nl=20,
             r_tol=1e-10),
        # a dozen uneven mass-matrix solves advanced together
        dict(name="batch-w0-12", kind="batch", space="w0", count=12, n_lo=12, n_hi=48, nl_lo=10,
             nl_hi=70, mix=3, r_tol=1e-10),
        # six uneven Helmholtz solves with the column preconditioner
        dict(name="batch-w2-6", kind="batch", space="w2", count=6, n_lo=12, n_hi=64, nl_lo=20,
             nl_hi=70, mix=4, r_tol=1e-10),
        # the FP64 mass matrix applied to a field, on its own
        dict(name="apply-w0-c48x30-f64", kind="apply", space="w0", n=48, nl=30, bits=64),
        # divergence and its transpose, W2 -> W3 -> W2, high columns
        dict(name="div-c48x70", kind="div", n=48, nl=70, bits=64),
        # one Arnoldi step of a caller's own solver over FP32 fields: apply,
        # preconditioner, and the vector procedures one by one
        dict(name="arnoldi-w2-c24x20-f32", kind="arnoldi", n=24, nl=20, basis=4, bits=32),
    ]


def _between(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["cg", "cg", "bicgstab", "gmres", "refined", "mrhs", "batch", "apply", "div",
                       "arnoldi"])
    tol = round(10.0 ** rng.uniform(-10, -8), 13)
    nl = _between(rng, 3, 70)
    # columns up to the cell counts of the listed cases
    wide = min(96, int(math.sqrt(96 * 96 * 30 / nl)))
    if kind == "cg":
        return dict(kind="solve", method="cg", n=_between(rng, 4, min(48, wide)), nl=nl, r_tol=tol)
    if kind == "bicgstab":
        return dict(kind="solve", method=kind, n=_between(rng, 4, min(64, wide)), nl=nl, r_tol=tol)
    if kind in ("gmres", "refined"):
        return dict(kind="solve", method=kind, n=_between(rng, 8, wide), nl=nl, r_tol=1e-8)
    if kind == "mrhs":
        return dict(kind="mrhs", method=rng.choice(["cg", "cg", "block"]),
                    mma=rng.choice(["tf32", "bf16"]), n=_between(rng, 8, 40),
                    nl=rng.randint(6, 30), r_tol=1e-10)
    if kind == "batch":
        w0 = rng.random() < 0.5
        return dict(kind="batch", space="w0" if w0 else "w2", count=rng.randint(2, 6), n_lo=8,
                    n_hi=40, nl_lo=10, nl_hi=50, mix=rng.randrange(10 ** 6), r_tol=1e-10)
    if kind == "apply":
        return dict(kind="apply", space=rng.choice(["w0", "w2"]), n=_between(rng, 24, min(64, wide)),
                    nl=max(nl, 10), bits=rng.choice([32, 64]))
    if kind == "div":
        return dict(kind="div", n=_between(rng, 8, min(64, wide)), nl=nl, bits=rng.choice([32, 64]))
    return dict(kind="arnoldi", n=_between(rng, 4, min(64, wide)), nl=nl, basis=rng.randint(1, 8),
                bits=rng.choice([32, 64]))


# ------------------------------------------------------------------ inputs
def _space(case):
    if case["kind"] in ("solve",):
        return "w0" if case["method"] == "cg" else "w2"
    return {"mrhs": "w0", "div": "w2", "arnoldi": "w2"}.get(case["kind"]) or case["space"]


def _problem(case, seed, **more):
    """Mesh, dofmap and local matrices of the case, with its vertices perturbed
    by the seed: the arrays that a model hands to the package."""
    make = mg.w0_problem if _space(case) == "w0" else mg.w2_problem
    return make(case["n"], case["nl"], seed=seed % (1 << 20), **more)


def _normal(seed, k, *shape):
    return np.random.default_rng([seed, k]).standard_normal(shape)


def _specs(case, seed):
    """(n, nl, mesh seed, right-hand side seed) of a batch's systems."""
    r = random.Random(case["mix"])
    return [(r.randint(case["n_lo"], case["n_hi"]), r.randint(case["nl_lo"], case["nl_hi"]),
             (seed * 64 + i) % (1 << 30), (seed * 64 + i) % (1 << 30) + 7)
            for i in range(case["count"])]


class _Device:
    """A field's device array for torch to look at; torch keeps this object,
    and with it the field, for as long as the tensor lives."""

    def __init__(self, v):
        self.field = v
        self.__cuda_array_interface__ = dict(shape=(v.undf[0],), strides=None, version=3,
                                             typestr="<f%d" % (v.precision // 8),
                                             data=(v.device_ptr(), False))


def _view(v):
    return torch.as_tensor(_Device(v), device="cuda")


def _bits(case):
    return lfx.R32 if case["bits"] == 32 else lfx.R64


def _divergence(ctx, p, bits):
    """The W2 -> W3 divergence as an operator of its own."""
    npc, cic = p.mesh.colour_lookup()
    return lfx.LmaOperator(ctx, p.ncell_2d, p.nlayers, 1, 6, p.extra["map_w3"], p.map,
                           p.extra["undf_w3"], p.undf, p.extra["div"], npc, cic, precision=bits)


def prepare(case, seed):
    ctx, kind = _ctx(), case["kind"]
    if kind == "batch":
        systems, xs = [], []
        for n, nl, ms, rs in _specs(case, seed):
            systems.append(wl.batch_system(ctx, n, nl, ms, mg.W0 if case["space"] == "w0" else mg.W2,
                                           rhs_seed=rs))
            xs.append(lfx.FieldVector(ctx, [systems[-1].undf]))
        b = lfx.Batch(ctx, 8 if case["space"] == "w0" else 6, len(systems), reserve_bytes=2 << 30)
        return dict(kind=kind, tol=case["r_tol"], batch=b, systems=systems, x=xs,
                    out=[_view(x) for x in xs])
    if kind == "div":
        p = _problem(case, seed, keep_parts=True)
        d = _divergence(ctx, p, _bits(case))
        u = lfx.FieldVector.from_array(ctx, _normal(seed, 1, p.undf), _bits(case))
        w3 = lfx.FieldVector(ctx, [p.extra["undf_w3"]], _bits(case))
        w2 = lfx.FieldVector(ctx, [p.undf], _bits(case))
        return dict(kind=kind, op=d, u=u, w3=w3, w2=w2, out=[_view(w3), _view(w2)])
    p = _problem(case, seed)
    if kind == "apply":
        op = wl._lma(ctx, p, _bits(case))
        x = lfx.FieldVector.from_array(ctx, _normal(seed, 1, p.undf), _bits(case))
        y = lfx.FieldVector(ctx, [p.undf], _bits(case))
        return dict(kind=kind, op=op, x=x, y=y, out=_view(y))
    if kind == "arnoldi":
        s = wl.device_w2(ctx, p, _bits(case))
        vs = _normal(seed, 1, case["basis"], p.undf) / math.sqrt(p.undf)
        basis = [lfx.FieldVector.from_array(ctx, v, _bits(case)) for v in vs]
        t, w = (lfx.FieldVector(ctx, [p.undf], _bits(case)) for _ in range(2))
        return dict(kind=kind, sys=s, basis=basis, t=t, w=w, out=_view(w))
    if kind == "mrhs":
        s = wl.device_w0(ctx, p)
        m = lfx.MultiRhsOperator(s.op, lfx.MRHS_BF16 if case["mma"] == "bf16" else lfx.MRHS_TF32, 64)
        m.autotune(3)
        b = torch.from_numpy(_normal(seed, 1, 64, p.undf)).cuda()
        method = lfx.MRHS_BLOCK_CG if case["method"] == "block" else lfx.MRHS_PER_RHS_CG
        st = torch.cuda.ExternalStream(ctx.stream)
        torch.cuda.synchronize()
        return dict(kind=kind, sys=s, m=m, b=b, x=torch.zeros_like(b), undf=p.undf, method=method,
                    tol=case["r_tol"], stream=st)
    # one solve; the large GMRES operators are tuned once, as the benchmark does
    method, tol = case["method"], case["r_tol"]
    if method == "cg":
        s = wl.device_w0(ctx, p)
        solver = lfx.ConjugateGradient(s.op, s.prec, tol, 1e-16, 5000)
    elif method == "bicgstab":
        s = wl.device_w2(ctx, p)
        solver = lfx.BiCGStab(s.op, s.prec, tol, 1e-16, 2000)
    else:
        s = wl.device_w2(ctx, p, lfx.R32 if method == "refined" else lfx.R64)
        s.op64.autotune(10)
        if method == "refined":
            s.op.autotune(10)
            solver = wl.refined_gmres(s, gcrk=10, inner_rtol=1e-4, r_tol=tol)
        else:
            solver = lfx.GMRES(s.op, s.prec, 10, tol, 1e-16, 200)
    x = lfx.FieldVector(ctx, [p.undf])
    return dict(kind=kind, sys=s, solver=solver, x=x, b=lfx.FieldVector.from_array(ctx, p.rhs),
                out=_view(x))


# ------------------------------------------------------------------ one pass
def run(s):
    kind = s["kind"]
    if kind == "solve":
        s["x"].set_scalar(0.0)
        s["solver"].apply(s["x"], s["b"])
        return s["out"]
    if kind == "mrhs":
        with torch.cuda.stream(s["stream"]):
            s["x"].zero_()
        s["m"].solve(s["sys"].op, s["sys"].diag, s["b"].data_ptr(), s["x"].data_ptr(), s["undf"],
                     r_tol=s["tol"], method=s["method"])
        return s["x"]
    if kind == "batch":
        b, slots = s["batch"], []
        for q, x in zip(s["systems"], s["x"]):
            x.set_scalar(0.0)
            slots.append(b.admit(q.ops[lfx.R64], q.ops[lfx.R32], q.prec32, q.b, x, s["tol"]))
        while b.step() < len(slots):
            pass
        for slot in slots:
            b.retire(slot)
        return s["out"]
    if kind == "apply":
        s["op"].apply(s["x"], s["y"])
        return s["out"]
    if kind == "div":
        s["op"].apply(s["u"], s["w3"])
        s["op"].apply_transpose(s["w3"], s["w2"])
        return s["out"]
    t, w = s["t"], s["w"]
    s["sys"].op.apply(s["basis"][-1], t)
    s["sys"].prec.apply(t, w)
    h = []
    for v in s["basis"]:
        h.append(w.dot(v))
        w.axpy(-h[-1], v)
    h.append(w.norm())
    w.scale(1.0 / h[-1])
    return [s["out"], np.array(h, dtype=np.float32)]


# ------------------------------------------------------------------ work
def _sizes(space, n, nl):
    """cells, dofs and entries of a cell's symmetric local matrix"""
    cells = 6 * n * n * nl
    if space == "w0":
        return cells, (6 * n * n + 2) * (nl + 1), 36
    return cells, 12 * n * n * nl + 6 * n * n * (nl + 1), 21


def _iterations(method, n, nl, tol):
    """About how many applies a solve takes (fitted to these problems)."""
    digits = -math.log10(tol) / 8.0
    if method == "cg":  # W0, Jacobi: grows with the smaller of width and height
        return 8.0 * min(n, 2.2 * nl) * digits + 10
    return 20.0 * digits  # W2 with the column preconditioner


def work(case):
    """The matrix (its symmetric half) once an iteration with one vector in and
    one out; right-hand side and solution once."""
    kind = case["kind"]
    if kind == "batch":
        total = dict(bytes=0.0, flops=0.0)
        for n, nl, _, _ in _specs(case, 0):
            cells, undf, half = _sizes(case["space"], n, nl)
            its = _iterations("cg" if case["space"] == "w0" else "pcg", n, nl, case["r_tol"])
            total["bytes"] += its * (cells * half * 4 + 2 * undf * 4) + 2 * undf * 8
            total["flops"] += its * (cells * half * 4 + 10 * undf)
        return total
    cells, undf, half = _sizes(_space(case), case["n"], case["nl"])
    if kind == "solve":
        size = 4 if case["method"] == "refined" else 8
        its = _iterations(case["method"], case["n"], case["nl"], case["r_tol"])
        return dict(bytes=its * (cells * half + 2 * undf) * size + 2 * undf * 8,
                    flops=its * (cells * half * 4 + 10 * undf))
    if kind == "mrhs":
        its = _iterations("cg", case["n"], case["nl"], case["r_tol"])
        size = 2 if case["mma"] == "bf16" else 4
        return dict(bytes=its * (cells * half * size + 2 * undf * 64 * 4) + 2 * undf * 64 * 8,
                    flops=its * 64 * (cells * half * 4 + 10 * undf))
    size = case["bits"] // 8
    if kind == "apply":
        return dict(bytes=(cells * half + 2 * undf) * size, flops=4.0 * cells * half)
    if kind == "div":
        return dict(bytes=(2 * cells * 6 + 2 * undf + cells) * size, flops=24.0 * cells)
    return dict(bytes=(cells * half + (case["basis"] + 2) * undf) * size,
                flops=4.0 * cells * half + (4 * case["basis"] + 8) * undf)


# ------------------------------------------------------------------ 64 bits
def _csr(p):
    """The assembled matrix of a problem's local matrices, FP64, by torch."""
    ndf, nl, dev = p.ndf, p.nlayers, "cuda"
    m = torch.from_numpy(np.ascontiguousarray(p.map)).to(dev).long() - 1
    dof = (m[:, None, :] + torch.arange(nl, device=dev)[None, :, None]).reshape(-1, ndf)
    a = torch.from_numpy(p.lma).to(dev).reshape(ndf, ndf, -1)  # [df2][df][cell level]
    out = None
    for i in range(ndf):
        at = torch.stack([dof[:, i].repeat(ndf), dof.t().reshape(-1)])
        part = torch.sparse_coo_tensor(at, a[:, i, :].reshape(-1), (p.undf, p.undf)).coalesce()
        out = part if out is None else (out + part).coalesce()
    return out.to_sparse_csr(), dof, a


def _diagonal(dof, a, undf):
    d = torch.zeros(undf, dtype=torch.float64, device="cuda")
    for i in range(dof.shape[1]):
        d.index_add_(0, dof[:, i], a[i, i])
    return d


def _solved(p, b):
    """A^-1 b by Jacobi CG in 64 bits, to far below any case's tolerance."""
    m, dof, a = _csr(p)
    d = _diagonal(dof, a, p.undf)
    del dof, a
    d = d if b.dim() == 1 else d[:, None]
    x = torch.zeros_like(b)
    r = b.clone()
    z = r / d
    q = z.clone()
    rz, start = (r * z).sum(0), (b * b).sum(0)
    for k in range(20000):
        y = m @ q
        alpha = rz / (q * y).sum(0)
        x += alpha * q
        r -= alpha * y
        z = r / d
        new = (r * z).sum(0)
        if k % 10 == 0 and bool(((r * r).sum(0) <= 1e-26 * start).all()):
            break
        q = z + (new / rz) * q
        rz = new
    return x


def _precondition(p, dof, a, r):
    """Column tridiagonal solve on the vertical faces, diagonal elsewhere."""
    z = r / _diagonal(dof, a, p.undf)
    nl, nc = p.nlayers, p.ncell_2d
    base = torch.from_numpy(np.ascontiguousarray(p.map[:, 4])).cuda().long() - 1
    rows = base[:, None] + torch.arange(nl + 1, device="cuda")[None, :]
    blk = {(i, j): a[j, i].reshape(nc, nl) for i in (4, 5) for j in (4, 5)}
    diag = torch.zeros(nc, nl + 1, dtype=torch.float64, device="cuda")
    diag[:, :nl] += blk[4, 4]
    diag[:, 1:] += blk[5, 5]
    up, low = blk[4, 5], blk[5, 4]
    f = r[rows]
    c, d = [], []
    for k in range(nl + 1):
        den = diag[:, k] if k == 0 else diag[:, k] - low[:, k - 1] * c[-1]
        d.append((f[:, k] if k == 0 else f[:, k] - low[:, k - 1] * d[-1]) / den)
        c.append(up[:, k] / den if k < nl else None)
    for k in range(nl - 1, -1, -1):
        d[k] = d[k] - c[k] * d[k + 1]
    z[rows.reshape(-1)] = torch.stack(d, 1).reshape(-1)
    return z


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        xs = []
        for n, nl, ms, rs in _specs(case, seed):
            p = (mg.w0_problem if case["space"] == "w0" else mg.w2_problem)(n, nl, seed=ms)
            rhs = (mg.uniform if case["space"] == "w0" else mg.normal)(rs, p.undf)
            xs.append(_solved(p, torch.from_numpy(rhs).cuda()))
        return xs
    p = _problem(case, seed, **({"keep_parts": True} if kind == "div" else {}))
    if kind == "solve":
        return _solved(p, torch.from_numpy(p.rhs).cuda())
    if kind == "mrhs":
        b = torch.from_numpy(_normal(seed, 1, 64, p.undf)).cuda()
        return _solved(p, b.t().contiguous()).t().contiguous()
    rounded = (lambda v: torch.from_numpy(v.astype(np.float32 if case["bits"] == 32 else np.float64))
               .cuda().double())
    if kind == "div":
        m = torch.from_numpy(np.ascontiguousarray(p.map)).cuda().long() - 1
        dof = (m[:, None, :] + torch.arange(p.nlayers, device="cuda")[None, :, None]).reshape(-1, 6)
        d = torch.from_numpy(p.extra["div"]).cuda().reshape(6, -1).t()
        m3 = torch.from_numpy(np.ascontiguousarray(p.extra["map_w3"])).cuda().long().reshape(-1) - 1
        at = (m3[:, None] + torch.arange(p.nlayers, device="cuda")[None, :]).reshape(-1)
        w3 = torch.zeros(p.extra["undf_w3"], dtype=torch.float64, device="cuda")
        w3[at] = (d * rounded(_normal(seed, 1, p.undf))[dof]).sum(1)
        w2 = torch.zeros(p.undf, dtype=torch.float64, device="cuda")
        w2.index_add_(0, dof.reshape(-1), (d * w3[at][:, None]).reshape(-1))
        return [w3, w2]
    m, dof, a = _csr(p)
    if kind == "apply":
        return m @ rounded(_normal(seed, 1, p.undf))
    vs = rounded(_normal(seed, 1, case["basis"], p.undf) / math.sqrt(p.undf))
    w = _precondition(p, dof, a, m @ vs[-1])
    h = []
    for v in vs:
        h.append(float(w @ v))
        w = w - h[-1] * v
    h.append(float(w.norm()))
    return [w / h[-1], np.array(h)]
