"""The engine's work as a user's program has it done, for timing.

Every case goes through the public Python interface (race_gb300.interface,
race_gb300.tuner): the matrix is ordered and registered once in prepare(),
run() is one call of the registered work with the operands in place. Inputs
come from the seed, generated on the GPU with the value distributions of
race_gb300.matgen:

power  y_k = A^k x, k = 1..p (RACE's matrix power), FP64/FP32/BF16 values;
batch  the block matrix power of many 2D stencils with several right-hand
       sides each, one persistent launch replayed from its CUDA graph;
sweep  one colored kernel call: SpMV, SpMTV, SymmSpMV (b zeroed, then
       accumulated), a symmetric Gauss-Seidel sweep or a Kaczmarz sweep
       (forward + backward each);
solve  FP64 iterative refinement to 1e-10 around symmetric Gauss-Seidel
       sweeps with FP64, FP32 or BF16 values;
mlp    loss and gradients of the tuner's network on one minibatch, or its
       predictions.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from race_gb300 import interface as ri
from race_gb300 import tuner

# values -> (matrix value type, vector type of sweeps and blocks)
TYPES = {"f64": (torch.float64, torch.float64), "f32": (torch.float32, torch.float32),
         "bf16": (torch.bfloat16, torch.float32)}
KERNELS = {"spmv": ri.SPMV, "spmtv": ri.SPMTV, "symmspmv": ri.SYMMSPMV, "gs": ri.GS, "kacz": ri.KACZ}
MLP_FEATURES = 34
PLAW_DEGREE = 12.5   # off-diagonal entries a row of the power-law graph on average, duplicates removed
SOLVE_STEPS = 20     # refinements of a solve, about
DEV = "cuda"


def listed():
    return [
        # the headline configuration: the matrix (669 MB) is far larger than the L2
        {"name": "power_st27_128_p8_f64", "kind": "power", "graph": "st27", "nx": 128, "ny": 128, "nz": 128,
         "power": 8, "values": "f64"},
        # the same operator with FP32 values on an ordinary, odd-sided domain
        {"name": "power_st27_97x113x89_p8_f32", "kind": "power", "graph": "st27", "nx": 97, "ny": 113, "nz": 89,
         "power": 8, "values": "f32"},
        # a small Laplacian that fits the L2 many times over: launches and latency count
        {"name": "power_lap7_32_p4_f64", "kind": "power", "graph": "lap7", "nx": 32, "ny": 32, "nz": 32,
         "power": 4, "values": "f64"},
        # a graph with hub rows and few levels, lowest-precision storage
        {"name": "power_plaw_150k_p4_bf16", "kind": "power", "graph": "plaw", "n": 150001, "power": 4,
         "values": "bf16"},
        # the reference's SymmSpMV on the 32^3 Laplacian: the smallest colored call
        {"name": "symmspmv_lap7_32_f64", "kind": "sweep", "kernel": "symmspmv", "graph": "lap7", "nx": 32, "ny": 32,
         "nz": 32, "threads": 1024, "dist": 2, "values": "f64"},
        # SymmSpMV of an ordinary 27-point operator, matrix larger than the L2
        {"name": "symmspmv_st27_95x87x91_f64", "kind": "sweep", "kernel": "symmspmv", "graph": "st27", "nx": 95,
         "ny": 87, "nz": 91, "threads": 256, "dist": 2, "values": "f64"},
        # symmetric Gauss-Seidel smoothing of a stencil operator
        {"name": "gs_st27_40x44x41_f64", "kind": "sweep", "kernel": "gs", "graph": "st27", "nx": 40, "ny": 44,
         "nz": 41, "threads": 256, "dist": 1, "values": "f64"},
        # Kaczmarz sweeps of an anisotropic 2D operator
        {"name": "kacz_aniso9_211x197_f64", "kind": "sweep", "kernel": "kacz", "graph": "aniso9", "nx": 211,
         "ny": 197, "nz": 1, "threads": 256, "dist": 2, "values": "f64"},
        # mixed-precision solve of a power-law system with hub rows
        {"name": "solve_plaw_100k_f32", "kind": "solve", "graph": "plaw", "n": 100003, "threads": 1024, "dist": 2,
         "values": "f32"},
        # many matrices of uneven size with 16 right-hand sides in one launch
        {"name": "batch_16_rhs16_p4_f64", "kind": "batch", "count": 16, "lo": 100, "hi": 700, "shapes": 1, "rhs": 16,
         "power": 4, "values": "f64"},
        {"name": "batch_24_rhs8_p4_f32", "kind": "batch", "count": 24, "lo": 100, "hi": 500, "shapes": 2, "rhs": 8,
         "power": 4, "values": "f32"},
        # one minibatch of the tuner's training (the batch of its committed searches)
        {"name": "mlp_grad_239", "kind": "mlp", "batch": 239, "grad": True},
    ]


def _loguni(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _sides(rng, graph, n):
    """Uneven grid sides with about n points in all."""
    if graph in ("aniso5", "aniso9"):
        r = math.exp(rng.uniform(-0.4, 0.4))
        return {"nx": max(3, round(math.sqrt(n) * r)), "ny": max(3, round(math.sqrt(n) / r)), "nz": 1}
    a, b = math.exp(rng.uniform(-0.3, 0.3)), math.exp(rng.uniform(-0.3, 0.3))
    s = n ** (1 / 3)
    return {"nx": max(3, round(s * a)), "ny": max(3, round(s * b)), "nz": max(3, round(s / (a * b)))}


def draw(rng):
    kind = rng.choice(["power", "power", "sweep", "sweep", "solve", "batch", "mlp"])
    values = rng.choice(["f64", "f64", "f32", "bf16"])
    if kind == "power":
        graph = rng.choice(["st27", "lap7", "plaw"])
        case = {"kind": kind, "graph": graph, "power": rng.randint(1, 8), "values": values}
        if graph == "plaw":
            return {**case, "n": _loguni(rng, 4000, 300000)}
        return {**case, **_sides(rng, graph, _loguni(rng, 4000, 1900000))}
    if kind == "sweep":
        kernel = rng.choice(["symmspmv", "symmspmv", "gs", "gs", "kacz", "spmv", "spmtv"])
        graph = rng.choice(["st27", "lap7", "aniso5", "aniso9", "plaw"])
        dist = rng.choice([1, 2]) if kernel in ("gs", "spmv") else 2
        case = {"kind": kind, "kernel": kernel, "graph": graph, "threads": rng.choice([64, 256, 1024]), "dist": dist,
                "values": values}
        top = 700000 if kernel in ("symmspmv", "spmv", "spmtv") and graph != "plaw" else 90000
        n = _loguni(rng, 4000, top)
        return {**case, "n": n} if graph == "plaw" else {**case, **_sides(rng, graph, n)}
    if kind == "solve":
        return {"kind": kind, "graph": "plaw", "n": _loguni(rng, 6000, 40000 if values == "f64" else 100000),
                "threads": rng.choice([64, 256, 1024]), "dist": 2, "values": values}
    if kind == "batch":
        lo = rng.randint(60, 140)
        return {"kind": kind, "count": rng.randint(1, 16), "lo": lo, "hi": lo + rng.randint(50, 450),
                "shapes": rng.randrange(1000), "rhs": rng.choice([1, 4, 8, 16, 32]) if values != "f64" else
                rng.choice([1, 4, 8, 16]), "power": rng.randint(2, 4), "values": values}
    return {"kind": kind, "batch": _loguni(rng, 37, 8000), "grad": rng.random() < 0.75}


# ---------------------------------------------------------------- inputs
def _gen(seed, k=0):
    g = torch.Generator(device=DEV)
    g.manual_seed(1000003 * int(seed) + k)
    return g


def _rand(shape, gen, lo=-1.0, hi=1.0):
    return lo + (hi - lo) * torch.rand(shape, dtype=torch.float64, device=DEV, generator=gen)


def _offsets(graph):
    """Positive half of the stencil as (dx, dy, dz)."""
    full = [(dx, dy, dz) for dz in (-1, 0, 1) for dy in (-1, 0, 1) for dx in (-1, 0, 1)]
    half = full[14:]
    if graph == "st27":
        return half
    if graph == "lap7":
        return [o for o in half if sum(map(abs, o)) == 1]
    flat = [o for o in half if o[2] == 0]
    return flat if graph == "aniso9" else [o for o in flat if sum(map(abs, o)) == 1]


def _stencil(graph, nx, ny, nz, gen, ratio=None):
    """Stencil matrix (row offsets, columns, values), the diagonal first in
    each row, the other columns ascending."""
    n = nx * ny * nz
    i = torch.arange(n, device=DEV)
    x, y, z = i % nx, (i // nx) % ny, i // (nx * ny)
    if ratio is None:
        ratio = math.exp(float(torch.rand(1, generator=gen, device=DEV)) * math.log(100.0))
    up = []
    for dx, dy, dz in _offsets(graph):
        ok = (x + dx >= 0) & (x + dx < nx) & (y + dy >= 0) & (y + dy < ny) & (z + dz >= 0) & (z + dz < nz)
        if graph == "st27":
            v = -1.0 + torch.rand(n, dtype=torch.float64, device=DEV, generator=gen) * (1 - 2.0 ** -53)
        elif graph == "lap7":
            v = torch.full((n,), -1.0, dtype=torch.float64, device=DEV)
        else:
            c = 0.5 * math.sqrt(ratio) if dx and dy else (ratio if dy else 1.0)
            v = torch.full((n,), -c, dtype=torch.float64, device=DEV)
        up.append((dx + nx * (dy + ny * dz), ok, v))
    cols, oks, vals = [i], [torch.ones(n, dtype=torch.bool, device=DEV)], [None]
    for off, ok, v in reversed(up):  # entries below the diagonal, mirrored
        cols.append(i - off)
        oks.append(torch.roll(ok, off))
        vals.append(torch.roll(v, off))
    for off, ok, v in up:
        cols.append(i + off)
        oks.append(ok)
        vals.append(v)
    ok = torch.stack(oks, 1)
    vals[0] = torch.zeros(n, dtype=torch.float64, device=DEV)
    val = torch.stack(vals, 1)
    if graph == "lap7":
        val[:, 0] = 6.0
    else:
        val[:, 0] = (val.abs() * ok).sum(1) + (1.0 if graph == "st27" else 1e-3)
    rp = torch.zeros(n + 1, dtype=torch.int32, device=DEV)
    rp[1:] = ok.sum(1).cumsum(0)
    return rp, torch.stack(cols, 1)[ok].to(torch.int32), val[ok]


def _powerlaw(n, gen):
    """Symmetric Chung-Lu graph, Pareto(2.1) weights with mean 16,
    off-diagonals N(0,1), diagonal = sum|off| + 1 first in each row."""
    w = (1.0 - torch.rand(n, dtype=torch.float64, device=DEV, generator=gen)) ** (-1.0 / 1.1)
    cdf = (w / w.sum()).cumsum(0)
    ends = torch.searchsorted(cdf, torch.rand((2, 8 * n), dtype=torch.float64, device=DEV, generator=gen))
    ends.clamp_(max=n - 1)
    a, b = ends.min(0).values, ends.max(0).values
    key = torch.unique((a * n + b)[a != b])
    a, b = key // n, key % n
    v = torch.randn(a.numel(), dtype=torch.float64, device=DEV, generator=gen)
    i = torch.arange(n, device=DEV)
    row, col, val = torch.cat([i, a, b]), torch.cat([i, b, a]), torch.cat([torch.ones_like(w), v, v])
    # sort key of an entry: its row, then the diagonal, then the column
    order = torch.argsort(row * (n + 1) + torch.where(col == row, 0, col + 1))
    row, col, val = row[order], col[order], val[order]
    rp = torch.zeros(n + 1, dtype=torch.int32, device=DEV)
    rp[1:] = torch.bincount(row, minlength=n).cumsum(0)
    val[rp[:-1].long()] = torch.segment_reduce(val.abs(), "sum", offsets=rp.long())
    return rp, col.to(torch.int32), val


def _matrix(case, gen):
    if case["graph"] == "plaw":
        return _powerlaw(case["n"], gen)
    return _stencil(case["graph"], case["nx"], case["ny"], case["nz"], gen)


def _permuted(rp, col, val, perm, inv):
    """The matrix in the engine's row order (entries keep their order)."""
    perm, inv = torch.as_tensor(perm, device=DEV).long(), torch.as_tensor(inv, device=DEV)
    lens = (rp[1:] - rp[:-1])[perm]
    rp2 = torch.zeros_like(rp)
    rp2[1:] = lens.cumsum(0)
    idx = torch.repeat_interleave(rp[:-1][perm] - rp2[:-1], lens) + torch.arange(col.numel(), device=DEV)
    return rp2, inv[col.long()[idx]], val[idx]


def _rows(rp):
    return torch.repeat_interleave(torch.arange(rp.numel() - 1, device=DEV), (rp[1:] - rp[:-1]).long())


def _upper(rp, col, val):
    rows = _rows(rp)
    keep = col >= rows
    rp2 = torch.zeros_like(rp)
    rp2[1:] = torch.bincount(rows[keep], minlength=rp.numel() - 1).cumsum(0)
    return rp2, col[keep].contiguous(), val[keep].contiguous()


def _product(rp, col, val, x):
    """A x with plain FP64 torch operations (x: n or n by right-hand sides)."""
    rows, out = _rows(rp), torch.zeros_like(x)
    step = 1 << 23
    for s in range(0, col.numel(), step):
        v, xc = val[s:s + step].double(), x[col[s:s + step].long()]
        out.index_add_(0, rows[s:s + step], v * xc if x.dim() == 1 else v[:, None] * xc)
    return out


def _level_order(graph, nx, ny, nz):
    """Row order of the matrix power on a grid: rows by distance from the
    corner row 0, ties in row order."""
    i = torch.arange(nx * ny * nz, device=DEV)
    x, y, z = i % nx, (i // nx) % ny, i // (nx * ny)
    far = x + y + z if graph in ("lap7", "aniso5") else torch.maximum(torch.maximum(x, y), z)
    return torch.sort(far, stable=True).indices


def _grids(case):
    """Shapes of a batch: sides, 5 or 9 points, coefficient ratio."""
    rng = np.random.Generator(np.random.PCG64(case["shapes"]))
    return [(int(rng.integers(case["lo"], case["hi"] + 1)), int(rng.integers(case["lo"], case["hi"] + 1)),
             "aniso5" if rng.random() < 0.5 else "aniso9", float(np.exp(rng.uniform(0.0, np.log(100.0)))))
            for _ in range(case["count"])]


def _engine(n, rp, col, threads, dist):
    return ri.Interface(n, threads, dist, rp.cpu().numpy(), col.cpu().numpy(), symm_hint=True)


def _ordered(case, gen):
    """A colored engine and the matrix in its order."""
    rp, col, val = _matrix(case, gen)
    rc = _engine(rp.numel() - 1, rp, col, case["threads"], case["dist"])
    assert rc.RACEColor() == 0
    return rc, _permuted(rp, col, val, rc.getPerm(), rc.getInvPerm())


def _mlp_data(case, seed):
    g = _gen(seed, 9)
    x = torch.randn((case["batch"], MLP_FEATURES), generator=g, device=DEV)
    return x, torch.randn((case["batch"], 1), generator=g, device=DEV)


# ---------------------------------------------------------------- the contract
def prepare(case, seed):
    kind = case["kind"]
    if kind == "mlp":
        x, t = _mlp_data(case, seed)
        return {"kind": kind, "net": tuner.Mlp(n_in=MLP_FEATURES, seed=int(seed)), "x": x, "t": t,
                "grad": case["grad"]}
    vt, xt = TYPES[case["values"]]
    gen = _gen(seed)
    if kind == "power":
        rp, col, val = _matrix(case, gen)
        n, p = rp.numel() - 1, case["power"]
        rc = _engine(n, rp, col, 1, ri.POWER)
        assert rc.RACEColor(p, 300e6) == 0
        perm = rc.getPerm()
        rp, col, val = _permuted(rp, col, val, perm, rc.getInvPerm())
        x = torch.zeros((p + 1) * n, dtype=torch.float64, device=DEV)
        x[:n] = _rand(n, _gen(seed, 1))[torch.as_tensor(perm, device=DEV).long()]
        fid = rc.registerFunction(ri.MPK, ri.Operands(ri.DeviceCsr(n, rp, col, val.to(vt)), x), power=p)
        assert fid >= 0
        return {"kind": kind, "rc": rc, "fid": fid, "x": x}
    if kind == "batch":
        batch, keep = ri.Batch(), []
        for i, (nx, ny, graph, ratio) in enumerate(_grids(case)):
            rp, col, val = _stencil(graph, nx, ny, 1, gen, ratio)
            n, p, m = nx * ny, case["power"], case["rhs"]
            rc = _engine(n, rp, col, 1, ri.POWER)
            assert rc.RACEColor(p, 256e6) == 0
            perm = rc.getPerm()
            rp, col, val = _permuted(rp, col, val, perm, rc.getInvPerm())
            x = torch.zeros((p + 1, n, m), dtype=xt, device=DEV)
            x[0] = _rand((n, m), _gen(seed, 10 + i)).to(xt)[torch.as_tensor(perm, device=DEV).long()]
            fid = rc.registerMpkBlock(ri.Operands(ri.DeviceCsr(n, rp, col, val.to(vt)), x), p, m)
            assert fid >= 0
            batch.add(rc, fid)
            keep.append((rc, x))
        batch.prepare()
        return {"kind": kind, "batch": batch, "keep": keep}
    rc, (rp, col, val) = _ordered(case, gen)
    n = rp.numel() - 1
    if kind == "sweep":
        if case["kernel"] == "symmspmv":
            rp, col, val = _upper(rp, col, val)
        x, b = _rand(n, _gen(seed, 1)).to(xt), _rand(n, _gen(seed, 2)).to(xt)
        fid = rc.registerFunction(KERNELS[case["kernel"]], ri.Operands(ri.DeviceCsr(n, rp, col, val.to(vt)), x, b))
        assert fid >= 0
        return {"kind": kind, "kernel": case["kernel"], "rc": rc, "fid": fid, "x": x, "b": b}
    # solve: the right-hand side of a known solution
    d, r = torch.zeros(n, dtype=xt, device=DEV), torch.zeros(n, dtype=xt, device=DEV)
    fid = rc.registerFunction(ri.GS, ri.Operands(ri.DeviceCsr(n, rp, col, val.to(vt)), d, r))
    assert fid >= 0
    m64, b = ri.DeviceCsr(n, rp, col, val), torch.zeros(n, dtype=torch.float64, device=DEV)
    rc.spmv_plain(m64, _rand(n, _gen(seed, 1)), b)
    return {"kind": kind, "rc": rc, "fid": fid, "m64": m64, "b": b,
            "x": torch.zeros(n, dtype=torch.float64, device=DEV)}


def run(state):
    kind = state["kind"]
    if kind == "power":
        assert state["rc"].executeFunctionAsync(state["fid"]) == 0
        return state["x"]
    if kind == "batch":
        state["batch"].graphLaunch()
        return [x for _, x in state["keep"]]
    if kind == "sweep":
        rc, fid = state["rc"], state["fid"]
        if state["kernel"] in ("gs", "kacz"):
            assert rc.executeFunctionAsync(fid) == 0
            assert rc.executeFunctionAsync(fid, True) == 0
            return state["x"]
        if state["kernel"] != "spmv":
            state["b"].zero_()
        assert rc.executeFunctionAsync(fid) == 0
        return state["b"]
    if kind == "solve":
        state["x"].zero_()
        steps, _ = state["rc"].symmGsIr(state["fid"], state["m64"], state["b"], state["x"], tol=1e-10, maxIter=300)
        return {"x": state["x"], "refinements": steps}
    if state["grad"]:
        loss, grad = state["net"].loss_grad(state["x"], state["t"])
        return {"loss": loss, "grad": grad}
    return state["net"].forward(state["x"])


def _shape(case):
    """Rows and stored entries of a case's matrix (about, for the power-law
    graph)."""
    if case["graph"] == "plaw":
        return case["n"], int(case["n"] * (1 + PLAW_DEGREE))
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    n = nx * ny * nz
    return n, n + 2 * sum((nx - abs(a)) * (ny - abs(b)) * (nz - abs(c)) for a, b, c in _offsets(case["graph"]))


def work(case):
    if case["kind"] == "mlp":
        dims, m = [MLP_FEATURES, 128, 128, 128, 1], case["batch"]
        par = sum((i + 1) * o for i, o in zip(dims, dims[1:]))
        mac = sum(i * o for i, o in zip(dims, dims[1:]))
        if not case["grad"]:
            return {"bytes": 4 * (par + m * (MLP_FEATURES + 1)), "flops": 2 * m * mac}
        return {"bytes": 4 * (2 * par + m * (MLP_FEATURES + 1)), "flops": 2 * m * (3 * mac - dims[0] * dims[1])}
    vs, xs = {"f64": (8, 8), "f32": (4, 4), "bf16": (2, 4)}[case["values"]]
    p = case.get("power", 1)
    if case["kind"] == "batch":
        got = {"bytes": 0, "flops": 0}
        for nx, ny, graph, _ in _grids(case):
            n, nnz = _shape({"graph": graph, "nx": nx, "ny": ny, "nz": 1})
            got["bytes"] += nnz * (vs + 4) + 4 * (n + 1) + (p + 1) * n * case["rhs"] * xs
            got["flops"] += 2 * nnz * p * case["rhs"]
        return got
    n, nnz = _shape(case)
    if case["kind"] == "power":
        return {"bytes": nnz * (vs + 4) + 4 * (n + 1) + (p + 1) * n * 8, "flops": 2 * nnz * p}
    if case["kind"] == "solve":
        sweep, residual = 2 * (nnz * (vs + 4) + 4 * n + 3 * n * xs), nnz * 12 + 4 * n + 24 * n
        return {"bytes": SOLVE_STEPS * (sweep + residual), "flops": SOLVE_STEPS * 6 * nnz}
    if case["kernel"] == "symmspmv":
        up = (nnz + n) // 2
        return {"bytes": up * (vs + 4) + 4 * (n + 1) + 2 * n * xs, "flops": 2 * nnz}
    if case["kernel"] in ("spmv", "spmtv"):
        return {"bytes": nnz * (vs + 4) + 4 * (n + 1) + 2 * n * xs, "flops": 2 * nnz}
    flops = 2 * nnz if case["kernel"] == "gs" else 6 * nnz
    return {"bytes": 2 * (nnz * (vs + 4) + 4 * (n + 1) + 3 * n * xs), "flops": 2 * flops}


def exact(case, seed):
    kind = case["kind"]
    if kind == "mlp":
        x, t = _mlp_data(case, seed)
        theta = torch.as_tensor(tuner.init_params(int(seed), MLP_FEATURES), device=DEV).double()
        dims, at, w = [MLP_FEATURES, 128, 128, 128, 1], 0, theta.clone().requires_grad_(case["grad"])
        h = x.double()
        for k, (i, o) in enumerate(zip(dims, dims[1:])):
            h = h @ w[at:at + i * o].view(o, i).T + w[at + i * o:at + i * o + o]
            at += i * o + o
            h = torch.relu(h) if k < 3 else h
        if not case["grad"]:
            return h
        loss = ((h - t.double()) ** 2).mean()
        loss.backward()
        return {"loss": float(loss), "grad": w.grad.cpu().numpy()}
    vt, xt = TYPES[case["values"]]
    gen = _gen(seed)
    if kind == "power" and case["graph"] != "plaw":
        rp, col, val = _matrix(case, gen)
        val = val.to(vt).double()
        order = _level_order(case["graph"], case["nx"], case["ny"], case["nz"])
        x, out = _rand(rp.numel() - 1, _gen(seed, 1)), []
        for _ in range(case["power"] + 1):
            out.append(x[order])
            x = _product(rp, col, val, x)
        return torch.cat(out)
    if kind == "batch":
        got = []
        for i, (nx, ny, graph, ratio) in enumerate(_grids(case)):
            rp, col, val = _stencil(graph, nx, ny, 1, gen, ratio)
            val, order = val.to(vt).double(), _level_order(graph, nx, ny, 1)
            x, out = _rand((nx * ny, case["rhs"]), _gen(seed, 10 + i)).to(xt).double(), []
            for _ in range(case["power"] + 1):
                out.append(x[order])
                x = _product(rp, col, val, x)
            got.append(torch.stack(out))
        return got
    if kind == "solve":
        return {"x": _rand(case["n"], _gen(seed, 1)), "refinements": None}
    return None  # the order of a coloring's rows, and of the power-law graph's, is the engine's own
