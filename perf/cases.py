"""The work this framework is used for, as cases that can be timed and checked: multigrid-preconditioned
PCG solves on the unit square and cube (one system, many right-hand sides, batches of uneven
instances, a parametric family assembled on the device), the LAFEM::Arch operations, and the warm-start
network's training and inference.

Every case is a dict of plain values with a "kind":
  pcg      one Poisson system, fixed matrix, new right-hand side         (PCG.correct_device)
  family   one instance of the parametric family: assembly, update, solve (ParametricFamily.setup/.solve)
  multi    32 or 64 right-hand sides of one system                       (MultiRhsPCG.solve_device)
  batch    independent instances of uneven level, kappa fields           (BatchPCG.solve_device)
  train    optimisation steps of the U-Net, parameters read back         (UNet.train_step/.get_params)
  infer    one prediction                                                (UNet.forward)
  ops      the operations of one Richardson-Jacobi step                  (arch.*)
"""
from __future__ import annotations

import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "feat3.doxytest_b200"))

import featb200 as fb  # noqa: E402
from featb200 import assembly as AS  # noqa: E402
from featb200.assembly_gpu import Q1Assembler2D  # noqa: E402
from featb200.unet import LAYERS, UNet, init_params  # noqa: E402
from featb200.warmstart import ParametricFamily  # noqa: E402

DEV = "cuda"
F64 = torch.float64
LR = 2e-3          # the learning rate that training starts with


def listed():
    return [
        # a small solve inside a larger program: everything is latency
        {"name": "pcg2d_l5_f64", "kind": "pcg", "dim": 2, "level": 5, "precision": "f64", "numbering": "grid",
         "cycle": "V", "sources": 8},
        # the plain method at the size of the reference's tutorial
        {"name": "pcg2d_l7_f64", "kind": "pcg", "dim": 2, "level": 7, "precision": "f64", "numbering": "grid",
         "cycle": "V", "sources": 8},
        # a caller with the reference's own vertex numbering (coarse vertices first), reordered by the solver
        {"name": "pcg2d_l9_f64_rcm", "kind": "pcg", "dim": 2, "level": 9, "precision": "f64", "numbering": "hierarchical",
         "cycle": "V", "sources": 8},
        # the flagship: a million unknowns, FP32 V-cycle inside FP64 PCG
        {"name": "pcg2d_l10_f32", "kind": "pcg", "dim": 2, "level": 10, "precision": "f32", "numbering": "grid",
         "cycle": "V", "sources": 8},
        # one system on the cube (27-point rows)
        {"name": "pcg3d_l6_f32", "kind": "pcg", "dim": 3, "level": 6, "precision": "f32", "numbering": "grid",
         "cycle": "V", "sources": 8},
        # generating one training instance: device assembly of all levels, new values, solve
        {"name": "family_l9_f64", "kind": "family", "level": 9, "precision": "f64", "instance": 0},
        # many load cases of one operator
        {"name": "multi2d_l8_k32_f64", "kind": "multi", "dim": 2, "level": 8, "rhs": 32, "precision": "f64", "sources": 8},
        {"name": "multi3d_l6_k64_f32", "kind": "multi", "dim": 3, "level": 6, "rhs": 64, "precision": "f32", "sources": 8},
        # many instances of uneven size with their own coefficients
        {"name": "batch64_l5to9_f32", "kind": "batch", "count": 64, "low": 5, "high": 9, "precision": "f32", "levels": 7,
         "sources": 8},
        # training steps of the warm-start network, and a prediction with it
        {"name": "train_g129_b32", "kind": "train", "grid": 129, "batch": 32, "steps": 4},
        {"name": "infer_g129_b1", "kind": "infer", "grid": 129, "batch": 1},
        # a solver of the reference that calls the operations one by one
        {"name": "ops_n263169_f64", "kind": "ops", "rows": 263169, "dtype": "f64", "ragged": False},
    ]


def draw(rng):
    kind = rng.choice(["pcg", "pcg", "pcg", "pcg", "family", "multi", "multi", "batch", "batch", "train", "infer", "ops"])
    prec = rng.choice(["f64", "f32", "f32", "f32_bf16"])
    if kind == "pcg":
        dim = rng.choice([2, 2, 2, 3])
        level = rng.randint(4, 10) if dim == 2 else rng.randint(3, 6)
        return {"kind": kind, "dim": dim, "level": level, "precision": prec,
                "numbering": rng.choice(["grid", "grid", "hierarchical"]), "cycle": rng.choice(["V", "V", "V", "F"]),
                "sources": rng.randint(1, 40)}
    if kind == "family":
        return {"kind": kind, "level": rng.randint(5, 9), "precision": rng.choice(["f64", "f32"]),
                "instance": rng.randint(1, 20000)}
    if kind == "multi":
        dim = rng.choice([2, 3])
        level = rng.randint(4, 8) if dim == 2 else rng.randint(3, 6)
        rhs = rng.choice([32, 64]) if (dim, level, prec) != (3, 6, "f64") else 32
        return {"kind": kind, "dim": dim, "level": level, "rhs": rhs, "precision": prec, "sources": rng.randint(1, 40)}
    if kind == "batch":
        low = rng.randint(3, 6)
        c = {"kind": kind, "count": int(round(math.exp(rng.uniform(math.log(3), math.log(64))))), "low": low,
             "high": rng.randint(low, 9), "precision": prec, "levels": rng.randint(0, 1 << 20),
             "sources": rng.randint(1, 40)}
        while sum(4 ** lv for lv in _batch_levels(c)) > 4000000:   # no more unknowns than the listed batch
            c["count"] -= 1
        return c
    if kind in ("train", "infer"):
        c = {"kind": kind, "grid": rng.choice([33, 65, 129]), "batch": int(round(math.exp(rng.uniform(0.0, math.log(32)))))}
        return dict(c, steps=rng.randint(1, 4)) if kind == "train" else c
    return {"kind": kind, "rows": int(round(math.exp(rng.uniform(math.log(500), math.log(1.1e6))))),
            "dtype": rng.choice(["f64", "f32"]), "ragged": rng.choice([False, True])}


# ---------------------------------------------------------------------------- problem data
@functools.lru_cache(maxsize=None)
def _grid_levels(dim, level):
    """The mesh hierarchy's matrices, filters and transfers (the same for every right-hand side)."""
    return AS.poisson_hierarchy(level, dim, rhs="sine")[0]


@functools.lru_cache(maxsize=None)
def _hierarchical(dim, level):
    """order[k] = lexicographic vertex at place k when a refinement numbers the coarser mesh's vertices first."""
    n = 2 ** level + 1
    idx = np.indices((n,) * dim).reshape(dim, -1)
    age = np.zeros(idx.shape[1], dtype=np.int64)          # the coarsest level whose mesh has the vertex
    for lv in range(level):
        age += np.any(idx % (1 << (level - lv)) != 0, axis=0)
    return np.argsort(age, kind="stable")


@functools.lru_cache(maxsize=None)
def _hierarchical_levels(dim, level):
    def permuted(m, rows, cols):
        return fb.SparseMatrixCSR.from_scipy(m.to_scipy()[rows][:, cols])

    out, lv = [], _grid_levels(dim, level)
    for d in lv:
        o = _hierarchical(dim, d["level"])
        place = np.empty(o.size, dtype=np.uint64)
        place[o] = np.arange(o.size, dtype=np.uint64)
        e = {"matrix": permuted(d["matrix"], o, o), "level": d["level"],
             "filter": fb.UnitFilter(np.sort(place[d["filter"].indices.astype(np.int64)]))}
        if "transfer" in d:
            c = _hierarchical(dim, d["level"] - 1)
            e["transfer"] = fb.Transfer(permuted(d["transfer"].get_mat_prol(), o, c),
                                        permuted(d["transfer"].get_mat_rest(), c, o))
        out.append(e)
    return out


def _load(dim, level, params):
    """Load vector of a sum of Gaussians (rows c_1..c_dim, w, a), boundary entries zero: the product of one 1D
    load vector per direction and Gaussian, 3-point Gauss rule (x fastest)."""
    N = 2 ** level
    h = 1.0 / N
    p = torch.tensor(params, dtype=F64, device=DEV)
    g = math.sqrt(0.6)
    xi = torch.tensor([-g, 0.0, g], dtype=F64, device=DEV)
    w = torch.tensor([5.0, 8.0, 5.0], dtype=F64, device=DEV) / 9.0
    xq = (torch.arange(N, dtype=F64, device=DEV)[:, None] + (1.0 + xi) / 2.0) * h
    lines = []
    for d in range(dim):
        f = torch.exp(-((xq[None] - p[:, d, None, None]) ** 2) / (2.0 * p[:, dim, None, None] ** 2)) * w * (h / 2.0)
        b = torch.zeros(p.shape[0], N + 1, dtype=F64, device=DEV)
        b[:, :-1] += (f * (1.0 - xi) / 2.0).sum(-1)
        b[:, 1:] += (f * (1.0 + xi) / 2.0).sum(-1)
        b[:, 0] = 0.0
        b[:, -1] = 0.0
        lines.append(b)
    a = p[:, dim + 1]
    if dim == 2:
        return torch.einsum("k,ky,kx->yx", a, lines[1], lines[0]).reshape(-1).contiguous()
    return torch.einsum("k,kz,ky,kx->zyx", a, lines[2], lines[1], lines[0]).reshape(-1).contiguous()


def _sources(case, seed):
    dim = case.get("dim", 2)
    return AS.gauss_params(seed, dim, case["sources"], (0.03, 0.12) if dim == 3 else (0.02, 0.1))


def _batch_levels(case):
    return [int(v) for v in np.random.default_rng(case["levels"]).integers(case["low"], case["high"] + 1, case["count"])]


def _batch_params(case, seed, k):
    return _sources(case, [seed, k, 0]), AS.field_params([seed, k, 1])


@functools.lru_cache(maxsize=None)
def _assembler(level):
    return Q1Assembler2D(level)


def _kappa_hierarchy(level, field):
    """A hierarchy whose matrices come from the device assembly, in host containers as the batch takes them."""
    levels = []
    for d in _grid_levels(2, level):
        asm = _assembler(d["level"])
        values, _ = asm.assemble(field, rhs=False)
        levels.append(dict(d, matrix=fb.SparseMatrixCSR(asm.row_ptr, asm.col_ind, values.cpu().numpy(), (asm.n, asm.n))))
    return fb.build_hierarchy(levels)


def _net_data(case, seed, count):
    """Inputs (f over its RMS, log kappa) and targets of unit size, as the warm start's training sees them."""
    gen = torch.Generator(device=DEV).manual_seed(int(seed))
    G = case["grid"]
    B = count * case["batch"]

    def rnd(*s):
        return torch.rand(*s, generator=gen, device=DEV)

    def normal(*s):
        return torch.randn(*s, generator=gen, device=DEV)

    t = torch.linspace(0, 1, G, device=DEV)
    c, w, a = 0.1 + 0.8 * rnd(B, 8, 2), 0.02 + 0.08 * rnd(B, 8), normal(B, 8)
    ex = torch.exp(-((t - c[:, :, :1]) ** 2) / (2 * w[:, :, None] ** 2))
    ey = torch.exp(-((t - c[:, :, 1:]) ** 2) / (2 * w[:, :, None] ** 2))
    f = torch.einsum("bk,bky,bkx->byx", a, ey, ex)
    f = f / f.pow(2).mean(dim=(1, 2), keepdim=True).sqrt()
    k = torch.arange(-8, 8, device=DEV, dtype=torch.float32)
    den = k[:, None] ** 2 + k[None, :] ** 2
    amp = torch.where(den > 0, 1.0 / den.clamp_min(1.0), torch.zeros_like(den))
    coef = torch.complex(normal(B, 16, 16), normal(B, 16, 16)) * amp / amp.pow(2).sum().sqrt()
    wave = torch.exp(2j * math.pi * k[:, None] * t[None, :])
    logk = torch.einsum("bij,ix,jy->byx", coef, wave, wave).real
    s = torch.sin(math.pi * torch.arange(1, 5, device=DEV)[:, None] * t[None, :])
    y = torch.einsum("bij,ix,jy->byx", normal(B, 4, 4) / 2.0, s, s)
    x = torch.stack([f, logk], dim=1).float().view(count, case["batch"], 2, G, G).contiguous()
    return x, y.float().view(count, case["batch"], G, G).contiguous()


def _ops_data(case, seed):
    """A row-sorted CSR matrix with the 9-point stencil of a grid of about sqrt(rows) columns (every third entry off the
    diagonal missing where ragged), dominant diagonal, and the vectors of a Jacobi step."""
    n = case["rows"]
    dt, it = (F64, torch.int64) if case["dtype"] == "f64" else (torch.float32, torch.int32)
    gen = torch.Generator(device=DEV).manual_seed(int(seed))
    W = max(3, int(round(math.sqrt(n))))
    off = torch.tensor([-W - 1, -W, -W + 1, -1, 0, 1, W - 1, W, W + 1], device=DEV)
    col = torch.arange(n, device=DEV)[:, None] + off
    keep = (col >= 0) & (col < n)
    if case["ragged"]:
        keep &= (torch.rand(n, 9, generator=gen, device=DEV) < 0.67) | (off == 0)
    val = torch.where(off == 0, 8.0, -1.0) + 0.5 * torch.rand(n, 9, generator=gen, device=DEV)
    rp = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    rp[1:] = keep.sum(1).cumsum(0)
    x, b = (torch.randn(n, generator=gen, device=DEV, dtype=F64).to(dt) for _ in range(2))
    idx = torch.arange(0, n, 129, device=DEV)
    return {"val": val[keep].to(dt).contiguous(), "col": col[keep].to(it).contiguous(), "rp": rp.to(it), "x": x, "b": b,
            "dinv": (0.7 / val[:, 4]).to(dt).contiguous(), "idx": idx.to(it)}


# ---------------------------------------------------------------------------- the interface
def prepare(case, seed):
    kind = case["kind"]
    if kind == "pcg":
        dim, level = case["dim"], case["level"]
        hier = case["numbering"] == "hierarchical"
        solver = fb.build_pcg_multigrid(_hierarchical_levels(dim, level) if hier else _grid_levels(dim, level),
                                        precision=case["precision"], ordering="rcm" if hier else "native",
                                        cycle=case["cycle"])
        b = _load(dim, level, _sources(case, seed))
        if hier:
            b = b[torch.tensor(_hierarchical(dim, level), device=DEV)].contiguous()
        return {"kind": kind, "solver": solver, "b": b, "x": torch.empty_like(b)}
    if kind == "family":
        fam = ParametricFamily(case["level"], max(3, case["level"] - 2), precision=case["precision"], seed_base=seed)
        return {"kind": kind, "family": fam, "instance": case["instance"], "x": torch.empty(fam.n, dtype=F64, device=DEV)}
    if kind == "multi":
        dim, level, K = case["dim"], case["level"], case["rhs"]
        solver = fb.MultiRhsPCG(fb.build_hierarchy(_grid_levels(dim, level)), K, precision=case["precision"])
        b = torch.stack([_load(dim, level, _sources(case, [seed, j])) for j in range(K)], dim=1)
        return {"kind": kind, "solver": solver, "b": b.contiguous(), "x": torch.empty_like(b)}
    if kind == "batch":
        levels = _batch_levels(case)
        params = [_batch_params(case, seed, k) for k in range(len(levels))]
        solver = fb.BatchPCG([_kappa_hierarchy(lv, f) for lv, (_, f) in zip(levels, params)], precision=case["precision"])
        b = torch.cat([_load(2, lv, g) for lv, (g, _) in zip(levels, params)])
        return {"kind": kind, "solver": solver, "b": b, "x": torch.empty_like(b)}
    if kind == "train":
        x, y = _net_data(case, seed, case["steps"])
        net = UNet(case["grid"], case["batch"], params=init_params(seed))
        return {"kind": kind, "net": net, "x": x, "y": y, "g": torch.empty_like(y[0])}
    if kind == "infer":
        x, _ = _net_data(case, seed, 1)
        return {"kind": kind, "net": UNet(case["grid"], case["batch"], params=init_params(seed)), "x": x[0]}
    d = _ops_data(case, seed)
    return dict(d, kind=kind, r=torch.empty_like(d["x"]), d=torch.empty_like(d["x"]), y=torch.empty_like(d["x"]))


def run(state):
    kind, x = state["kind"], state["x"]
    if kind == "pcg":
        x.zero_()
        state["solver"].correct_device(x, state["b"])
        return x
    if kind == "family":
        fam = state["family"]
        fam.setup(state["instance"])
        x.zero_()
        fam.solve(x)
        return x
    if kind in ("multi", "batch"):
        x.zero_()
        state["solver"].solve_device(x, state["b"])
        return x
    if kind == "train":
        net = state["net"]
        loss = [net.train_step(x[i], state["y"][i], LR, state["g"]).clone() for i in range(x.shape[0])]
        return {"loss": torch.cat(loss), "params": net.get_params()}
    if kind == "infer":
        return state["net"].forward(x)
    r, d, y = state["r"], state["d"], state["y"]
    n = r.numel()
    fb.arch.apply_csr(r, -1.0, x, 1.0, state["b"], state["val"], state["col"], state["rp"], n)
    fb.arch.unit_filter_def(r, state["idx"])
    fb.arch.component_product(d, state["dinv"], r)
    fb.arch.axpy(y, 1.0, d, x)
    return {"r": r, "d": d, "y": y, "dot": fb.arch.dot(r, d), "norm": fb.arch.norm2(r)}


ITERATIONS = 6     # of PCG to a relative residual of 1e-8, over these problems 5 to 9


def _solve_work(dim, level, precision, rhs=1):
    """One PCG iteration cannot do without: the FP64 matrix values once and five FP64 vectors' reads and writes;
    on every level the V-cycle's values twice (before and after the coarse correction), the transfers once each
    and six vectors, in the V-cycle's precision.  Per matrix value and right-hand side two operations; four
    smoothing steps, one defect and the transfers per level."""
    sv = {"f64": 8, "f32": 4, "f32_bf16": 2}[precision]
    sx = 8 if precision == "f64" else 4
    stencil, transfer = (9, 2.25) if dim == 2 else (27, 3.375)
    nbytes = flops = 0.0
    n = float(2 ** level + 1) ** dim
    nbytes += n * stencil * 8 + 10 * n * 8 * rhs
    flops += n * rhs * (2 * stencil + 12)
    for lv in range(level, 0, -1):
        n = float(2 ** lv + 1) ** dim
        nbytes += 2 * n * stencil * sv + 2 * n * transfer * sv + 6 * n * sx * rhs
        flops += n * rhs * (2 * stencil * 4 + 4 * transfer + 10)
    return ITERATIONS * nbytes, ITERATIONS * flops


def work(case):
    kind = case["kind"]
    if kind == "pcg":
        nbytes, flops = _solve_work(case["dim"], case["level"], case["precision"])
    elif kind == "family":
        nbytes, flops = _solve_work(2, case["level"], case["precision"])
        cells = 4.0 / 3.0 * 4 ** case["level"]
        nbytes, flops = nbytes + cells * 9 * 8, flops + cells * (9 * 16 * 4 + 16 * 9 * 2)
    elif kind == "multi":
        nbytes, flops = _solve_work(case["dim"], case["level"], case["precision"], case["rhs"])
    elif kind == "batch":
        each = [_solve_work(2, lv, case["precision"]) for lv in _batch_levels(case)]
        nbytes, flops = sum(e[0] for e in each), sum(e[1] for e in each)
    elif kind in ("train", "infer"):
        G = [case["grid"]]
        for _ in range(3):
            G.append((G[-1] + 1) // 2)
        at = [0, 1, 2, 3, 3, 3, 2, 1, 0, 0]
        macs = sum(9.0 * ci * co * G[g] ** 2 for (ci, co), g in zip(LAYERS, at))
        acts = sum(co * float(G[g]) ** 2 for (_, co), g in zip(LAYERS, at))
        if kind == "infer":
            return {"bytes": case["batch"] * (2 * acts * 2 + 12.0 * G[0] ** 2), "flops": case["batch"] * 2 * macs}
        # forward writes and reads the BF16 activations, backward reads them and moves their gradients
        nbytes = case["steps"] * case["batch"] * (6 * acts * 2 + 16.0 * G[0] ** 2)
        flops = case["steps"] * case["batch"] * 6 * macs
    else:
        n, s = case["rows"], 8 if case["dtype"] == "f64" else 4
        nnz = n * (9.0 if not case["ragged"] else 6.4)
        nbytes, flops = nnz * 2 * s + n * s * 12.0, nnz * 2 + n * 8.0
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    kind = case["kind"]
    if kind in ("pcg", "family", "multi", "batch"):
        # FP64: another order of the reductions moves these solutions by 1e-16, and by up to 1e-12 where the
        # coefficients are rough; FP32 V-cycles: the last bits of a preconditioner input move a solution by up to 2e-11
        return {"rel": 1e-12, "max": 1e-10} if case["precision"] == "f64" else {"rel": 5e-10, "max": 1e-8}
    if kind == "train":
        # BF16 operands: the parameters are 5e-3 to 8e-3 off the 64-bit ones, single ones by an Adam step's sign
        return {"rel": 1e-2, "max": 0.5}
    if kind == "infer":
        return {"rel": 1e-2, "max": 0.2}
    return {"rel": 1e-13, "max": 1e-10} if case["dtype"] == "f64" else {"rel": 1e-6, "max": 1e-4}


# ---------------------------------------------------------------------------- 64-bit results
def _poisson_exact(dim, level, b):
    """The Q1 Laplacian's inverse by its sine eigenvectors: b [n, columns], boundary entries zero."""
    N = 2 ** level
    j = torch.arange(1, N, dtype=F64, device=DEV)
    S = torch.sin(math.pi / N * j[:, None] * j[None, :]) * math.sqrt(2.0 / N)
    th = math.pi / N * j
    k, m = 2.0 * N * (1.0 - torch.cos(th)), (2.0 + torch.cos(th)) / (3.0 * N)
    B = b.reshape((N + 1,) * dim + (-1,))
    inner = (slice(1, N),) * dim
    v = B[inner]
    if dim == 2:
        lam = k[:, None] * m + m[:, None] * k
    else:
        lam = (k[:, None, None] * m[:, None] * m + m[:, None, None] * k[:, None] * m + m[:, None, None] * m[:, None] * k)
    for _ in range(2):
        for d in range(dim):
            v = torch.tensordot(S, v, dims=([1], [d])).movedim(0, d)
        if _ == 0:
            v = v / lam[..., None]
    out = torch.zeros_like(B)
    out[inner] = v
    return out.reshape(b.shape)


def _kappa_matrix(level, fields):
    """Element matrices of -div(kappa grad u) on every cell for each field: [fields, N, N, 4, 4], cells as (y, x)."""
    N = 2 ** level
    g = math.sqrt(0.6)
    xi = torch.tensor([-g, 0.0, g], dtype=F64, device=DEV)
    w = torch.tensor([5.0, 8.0, 5.0], dtype=F64, device=DEV) / 9.0
    t = ((torch.arange(N, dtype=F64, device=DEV)[:, None] + (1.0 + xi) / 2.0) / N).reshape(-1)
    sx = torch.tensor([-1.0, 1.0, -1.0, 1.0], dtype=F64, device=DEV)
    sy = torch.tensor([-1.0, -1.0, 1.0, 1.0], dtype=F64, device=DEV)
    gx = (sx * (1.0 + xi[:, None] * sy) / 4.0)[:, None].expand(3, 3, 4)      # [qy, qx, v]
    gy = (sy * (1.0 + xi[:, None] * sx) / 4.0)[None].expand(3, 3, 4)
    gg = (gx[..., :, None] * gx[..., None, :] + gy[..., :, None] * gy[..., None, :]) * (w[:, None] * w)[..., None, None]
    out = []
    for kx, ky, a, b, s in fields:
        kx, ky, a, b = (torch.tensor(np.asarray(v), dtype=F64, device=DEV) for v in (kx, ky, a, b))
        den = kx[:, None] ** 2 + ky ** 2
        c = torch.where(den > 0, torch.complex(a, -b) / den.clamp_min(1.0), torch.zeros_like(den) + 0j)
        ex, ey = (torch.exp(2j * math.pi * k[:, None] * t) for k in (kx, ky))
        kap = torch.exp(float(s) * torch.einsum("ij,jy,ix->yx", c, ey, ex).real).reshape(N, 3, N, 3)
        out.append(torch.einsum("yqxp,qpuv->yxuv", kap, gg))
    return torch.stack(out)


def _kappa_exact(level, fields, b):
    """Jacobi-preconditioned CG to the limit of 64 bits, all fields of one level together: b [fields, n]."""
    N = 2 ** level
    K = _kappa_matrix(level, fields)
    st = torch.zeros(len(fields), N + 1, N + 1, 3, 3, dtype=F64, device=DEV)   # the 9-point rows
    for u in range(4):
        for v in range(4):
            uy, ux, vy, vx = u >> 1, u & 1, v >> 1, v & 1
            st[:, uy:N + uy, ux:N + ux, 1 + vy - uy, 1 + vx - ux] += K[..., u, v]
    st = st[:, 1:N, 1:N]

    def apply(p):
        q = torch.zeros_like(p)
        s = sum(st[..., i, j] * p[:, i:N - 1 + i, j:N - 1 + j] for i in range(3) for j in range(3))
        q[:, 1:N, 1:N] = s
        return q

    dinv = torch.zeros(len(fields), N + 1, N + 1, dtype=F64, device=DEV)
    dinv[:, 1:N, 1:N] = 1.0 / st[..., 1, 1]
    r = b.reshape(-1, N + 1, N + 1).clone()
    x = torch.zeros_like(r)
    z = dinv * r
    p = z.clone()
    rz = (r * z).sum((1, 2), keepdim=True)
    stop = 1e-26 * rz
    for it in range(20 * (N + 1)):
        q = apply(p)
        al = rz / (p * q).sum((1, 2), keepdim=True).clamp_min(1e-300)
        x += al * p
        r -= al * q
        z = dinv * r
        new = (r * z).sum((1, 2), keepdim=True)
        if it % 50 == 49 and bool((new <= stop).all()):
            break
        p = z + (new / rz.clamp_min(1e-300)) * p
        rz = new
    return x.reshape(b.shape)


def _net_exact(params, x):
    """The network in 64 bits: params a flat tensor, x [B, 2, G, G]."""
    conv = torch.nn.functional.conv2d
    ws, at = [], 0
    for ci, co in LAYERS:
        w = params[at:at + co * 9 * ci].view(co, 3, 3, ci).permute(0, 3, 1, 2)
        ws.append((w, params[at + co * 9 * ci:at + co * 9 * ci + co]))
        at += co * 9 * ci + co

    def layer(i, v, dil=1):
        return conv(v, ws[i][0], ws[i][1], padding=dil, dilation=dil)

    def up(v):
        return torch.nn.functional.interpolate(v, size=2 * v.shape[-1] - 1, mode="bilinear", align_corners=True)

    e1 = layer(0, x).relu()
    e2 = layer(1, e1[..., ::2, ::2]).relu()
    e3 = layer(2, e2[..., ::2, ::2]).relu()
    e4 = layer(3, e3[..., ::2, ::2]).relu()
    e4 = layer(4, e4, 2).relu()
    e4 = layer(5, e4, 4).relu()
    d3 = layer(6, torch.cat([up(e4), e3], 1)).relu()
    d2 = layer(7, torch.cat([up(d3), e2], 1)).relu()
    d1 = layer(8, torch.cat([up(d2), e1], 1)).relu()
    return layer(9, d1)[:, 0]


def exact(case, seed):
    kind = case["kind"]
    if kind == "pcg":
        dim, level = case["dim"], case["level"]
        x = _poisson_exact(dim, level, _load(dim, level, _sources(case, seed))[:, None])[:, 0]
        return x[torch.tensor(_hierarchical(dim, level), device=DEV)] if case["numbering"] == "hierarchical" else x
    if kind == "multi":
        dim, level = case["dim"], case["level"]
        b = torch.stack([_load(dim, level, _sources(case, [seed, j])) for j in range(case["rhs"])], 1)
        return _poisson_exact(dim, level, b)
    if kind == "family":
        s = seed + 2 * case["instance"]
        return _kappa_exact(case["level"], [AS.field_params(s + 1)], _load(2, case["level"], AS.gauss_params(s, 2))[None])[0]
    if kind == "batch":
        levels = _batch_levels(case)
        out = [None] * len(levels)
        for lv in sorted(set(levels)):
            at = [k for k, v in enumerate(levels) if v == lv]
            for i in range(0, len(at), 8):
                ps = [_batch_params(case, seed, k) for k in at[i:i + 8]]
                x = _kappa_exact(lv, [f for _, f in ps], torch.stack([_load(2, lv, g) for g, _ in ps]))
                for k, v in zip(at[i:i + 8], x):
                    out[k] = v
        return torch.cat(out)
    if kind == "infer":
        x, _ = _net_data(case, seed, 1)
        with torch.no_grad():
            return _net_exact(torch.tensor(init_params(seed), dtype=F64, device=DEV), x[0].double())
    if kind == "train":
        x, y = _net_data(case, seed, case["steps"])
        p = torch.tensor(init_params(seed), dtype=F64, device=DEV)
        m, v, losses = torch.zeros_like(p), torch.zeros_like(p), []
        for t in range(case["steps"]):
            q = p.clone().requires_grad_(True)
            loss = (_net_exact(q, x[t].double()) - y[t].double()).square().mean()
            loss.backward()
            losses.append(loss.detach())
            m = 0.9 * m + 0.1 * q.grad
            v = 0.999 * v + 0.001 * q.grad ** 2
            p = p - LR * (m / (1 - 0.9 ** (t + 1))) / ((v / (1 - 0.999 ** (t + 1))).sqrt() + 1e-8)
        return {"loss": torch.stack(losses), "params": p}
    d = {k: (t.double() if t.is_floating_point() else t.long()) for k, t in _ops_data(case, seed).items()}
    rows = torch.repeat_interleave(torch.arange(case["rows"], device=DEV), d["rp"].diff())
    r = d["b"] - torch.zeros_like(d["x"]).index_add_(0, rows, d["val"] * d["x"][d["col"]])
    r[d["idx"]] = 0.0
    z = d["dinv"] * r
    return {"r": r, "d": z, "y": z + d["x"], "dot": (r * z).sum(), "norm": r.square().sum().sqrt()}
