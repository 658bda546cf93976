"""The measured work of this framework: calls of its public entry points as a
program that solves HPCG problems makes them.

Grids, tolerances and right-hand sides are those of the tests and of bench.py:
the 32^3 set, the 104^3 default local grid, the 128^3 differentiation problem,
16 uneven problems solved together, eight right-hand sides, a grid of several
tens of millions of rows. Right-hand sides are uniform on [-1, 1], the initial
guess is zero.

listed() and draw() give cases (dicts of plain values), prepare() the handle and
the vectors, run() one pass, work() the bytes and operations of one pass, and
exact() the same results in plain torch, in 64 bits.
"""
from __future__ import annotations

import math

import numpy as np
import torch

DEVICE = "cuda:0"


# ---- cases --------------------------------------------------------------------

def listed():
    return [
        # one operator product on the smallest test grid: a call's fixed cost
        dict(name="spmv_16", kind="spmv", nx=16, ny=16, nz=16),
        # one symmetric Gauss-Seidel step on a grid of odd sides
        dict(name="symgs_odd", kind="symgs", nx=75, ny=61, nz=53),
        # the vector routines of an iteration a user writes around the operators
        dict(name="vectors_2m", kind="vectors", n=2097153),
        # the FP64 preconditioner alone, 128^3
        dict(name="mg_128", kind="mg", nx=128, ny=128, nz=128),
        # the FP32 preconditioner alone, a small uneven grid
        dict(name="mg_f32_small", kind="mg_f32", nx=96, ny=64, nz=48),
        # the reference problem's grid, solved to the tolerance of the tests
        dict(name="cg_32", kind="cg", nx=32, ny=32, nz=32, max_iter=500, tol=1e-9, host=False),
        # the benchmark's default local grid from a C++ host: host vectors, a
        # fixed number of iterations
        dict(name="cg_host_104", kind="cg", nx=104, ny=104, nz=104, max_iter=30, tol=0.0, host=True),
        # the largest: tens of millions of rows, matrix far beyond the L2 cache
        dict(name="cg_384", kind="cg", nx=384, ny=384, nz=384, max_iter=12, tol=0.0, host=False),
        # the FP32 preconditioner inside FP64 flexible CG, to 1e-9
        dict(name="cg_mixed_160", kind="cg_mixed", nx=160, ny=160, nz=160, max_iter=500, tol=1e-9),
        # eight right-hand sides in lockstep
        dict(name="cg_multi_8", kind="cg_multi", nx=128, ny=128, nz=128, nrhs=8, max_iter=20, tol=0.0),
        # sixteen problems of uneven sizes solved together
        dict(name="batch_16", kind="batch", count=16, shape_seed=20251203, max_iter=500, tol=1e-9),
        # a training step: solve with given values, gradients of values and right-hand side
        dict(name="adjoint_128", kind="adjoint", nx=128, ny=128, nz=128, max_iter=500, tol=1e-10),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _sides(rng, lo, hi, step, max_rows):
    """Three sides in [lo, hi], multiples of step, of about the same size."""
    while True:
        base = math.exp(rng.uniform(math.log(lo), math.log(hi)))
        s = [min(hi, max(lo, int(round(base * rng.uniform(0.7, 1.4) / step)) * step)) for _ in range(3)]
        if s[0] * s[1] * s[2] <= max_rows:
            return dict(nx=s[0], ny=s[1], nz=s[2])


def draw(rng):
    kind = rng.choice(["spmv", "symgs", "vectors", "mg", "mg_f32", "cg", "cg_mixed", "cg_multi", "batch", "adjoint"])
    if kind == "vectors":
        return dict(kind=kind, n=_log_int(rng, 1000, 1 << 27))
    if kind in ("spmv", "symgs"):  # any sides (one level)
        return dict(kind=kind, **_sides(rng, 9, 256, 1, 256 ** 3))
    if kind in ("mg", "mg_f32"):  # four levels: sides are multiples of 8
        return dict(kind=kind, **_sides(rng, 16, 256, 8, 256 ** 3))
    if kind == "cg":
        s = _sides(rng, 16, 256, 8, 192 ** 3)
        if rng.random() < 0.5:
            return dict(kind=kind, **s, max_iter=500, tol=1e-9, host=rng.random() < 0.3)
        return dict(kind=kind, **s, max_iter=rng.randint(5, 30), tol=0.0, host=rng.random() < 0.3)
    if kind == "cg_mixed":
        return dict(kind=kind, **_sides(rng, 16, 192, 8, 160 ** 3), max_iter=500, tol=1e-9)
    if kind == "cg_multi":
        return dict(kind=kind, **_sides(rng, 16, 160, 8, 128 ** 3), nrhs=rng.randint(2, 8),
                    max_iter=rng.randint(5, 20), tol=0.0)
    if kind == "batch":
        return dict(kind=kind, count=rng.randint(4, 16), shape_seed=rng.randrange(1 << 30), max_iter=500, tol=1e-9)
    return dict(kind=kind, **_sides(rng, 16, 128, 8, 128 ** 3), max_iter=500, tol=1e-10)


def _dims(case):
    return case["nx"], case["ny"], case["nz"]


def _batch_dims(case):
    g = np.random.Generator(np.random.PCG64(case["shape_seed"]))
    return [tuple(int(v) for v in g.choice([32, 48, 64, 96, 128], 3)) for _ in range(case["count"])]


def _levels(case):
    """Operators alone take a one-level handle, as a grid of odd sides must."""
    return 1 if case["kind"] in ("spmv", "symgs") else 4


def _uniform(seed, stream, *shape):
    g = torch.Generator(device=DEVICE)
    g.manual_seed(int(seed) * 64 + stream)
    return torch.rand(*shape, generator=g, device=DEVICE, dtype=torch.float64) * 2.0 - 1.0


def _directions():
    return [(k // 9 - 1, (k // 3) % 3 - 1, k % 3 - 1) for k in range(27)]  # (sz, sy, sx) of slot k


def _span(n, s):
    return slice(max(0, -s), n - max(0, s)), slice(max(0, s), n - max(0, -s))


def _perturbed(dims, seed):
    """A seeded symmetric, strictly diagonally dominant 27-point matrix, [n, 27]
    by direction slot: off-diagonals -(1 + 0.1 u), diagonal 1.05 times the
    absolute sum of its row."""
    nx, ny, nz = dims
    v = torch.zeros(nz, ny, nx, 27, device=DEVICE, dtype=torch.float64)
    g = torch.Generator(device=DEVICE)
    for k, (sz, sy, sx) in enumerate(_directions()):
        if k <= 13:
            continue
        g.manual_seed(int(seed) * 64 + 32 + k)
        u = torch.rand(nz, ny, nx, generator=g, device=DEVICE, dtype=torch.float64) * 2.0 - 1.0
        (z0, z1), (y0, y1), (x0, x1) = _span(nz, sz), _span(ny, sy), _span(nx, sx)
        a = -(1.0 + 0.1 * u[z0, y0, x0])
        v[z0, y0, x0, k] = a
        v[z1, y1, x1, 26 - k] = a
    v[..., 13] = 1.05 * v.abs().sum(-1)
    return v.reshape(nx * ny * nz, 27)


# ---- a pass ---------------------------------------------------------------------

def prepare(case, seed):
    from hpcg_b200 import binding as B
    kind = case["kind"]
    if kind == "vectors":
        n = case["n"]
        return dict(case=case, lib=B, n=n, x=_uniform(seed, 0, n), y=_uniform(seed, 1, n),
                    w=torch.empty(n, device=DEVICE, dtype=torch.float64))
    if kind == "batch":
        dims = _batch_dims(case)
        b = [_uniform(seed, i, d[0] * d[1] * d[2]) for i, d in enumerate(dims)]
        return dict(case=case, batch=B.Batch(dims), b=b, x=[torch.empty_like(v) for v in b])
    dims = _dims(case)
    n = dims[0] * dims[1] * dims[2]
    s = dict(case=case, problem=B.Problem.generate(*dims, nlevels=_levels(case)))
    if kind == "cg_multi":
        s["b"] = _uniform(seed, 0, case["nrhs"], n)
    else:
        s["b"] = _uniform(seed, 0, n)
    s["x"] = torch.empty_like(s["b"])
    if kind == "symgs":
        s["x0"] = _uniform(seed, 1, n)
    if kind == "adjoint":
        s["values"] = _perturbed(dims, seed).requires_grad_(True)
        s["b"].requires_grad_(True)
        s["target"] = _uniform(seed, 1, n)
    if case.get("host"):
        s["b"], s["x"] = s["b"].cpu().numpy(), np.empty(n)
    return s


def run(s):
    c = s["case"]
    kind = c["kind"]
    if kind == "vectors":
        lib, n = s["lib"], s["n"]
        lib.ComputeWAXPBY(n, 1.0, s["x"], -0.75, s["y"], s["w"])
        return {"w": s["w"], "dot": lib.ComputeDotProduct(n, s["x"], s["w"]),
                "residual": lib.ComputeResidual(n, s["y"], s["w"])}
    if kind == "batch":
        for x in s["x"]:
            x.zero_()
        ni, nr, nr0 = s["batch"].CG_mixed(s["b"], s["x"], c["max_iter"], c["tol"])
        return {"x": s["x"], "iterations": ni, "normr": nr, "normr0": nr0}
    p = s["problem"]
    if kind == "spmv":
        p.ComputeSPMV(s["b"], s["x"])
        return {"y": s["x"]}
    if kind == "symgs":
        s["x"].copy_(s["x0"])
        p.ComputeSYMGS(s["b"], s["x"])
        return {"x": s["x"]}
    if kind == "mg":
        p.ComputeMG(s["b"], s["x"])
        return {"x": s["x"]}
    if kind == "mg_f32":
        p.ComputeMG_f32(s["b"], s["x"])
        return {"x": s["x"]}
    if kind == "adjoint":
        from hpcg_b200.autograd import HpcgSolve
        s["values"].grad = s["b"].grad = None
        x = HpcgSolve.apply(s["values"], s["b"], p, c["tol"], c["max_iter"])
        loss = 0.5 * (x - s["target"]).square().sum()
        loss.backward()
        return {"x": x, "grad_values": s["values"].grad, "grad_b": s["b"].grad}
    if c.get("host"):
        s["x"][:] = 0.0
    else:
        s["x"].zero_()
    if kind == "cg":
        ni, nr, nr0 = p.CG(s["b"], s["x"], c["max_iter"], c["tol"], True)
    elif kind == "cg_mixed":
        ni, nr, nr0 = p.CG_mixed(s["b"], s["x"], c["max_iter"], c["tol"])
    else:
        ni, nr, nr0 = p.CG_multi(s["b"], s["x"], c["max_iter"], c["tol"])
    return {"x": s["x"], "iterations": ni, "normr": nr, "normr0": nr0}


# ---- what a pass cannot do without ------------------------------------------------

# Slots a Gauss-Seidel sweep from x = 0 reads, of 27: the neighbours of colours
# already swept (13 on average) and the diagonal.
_FIRST = 14


def _vcycle(n, vb, nrhs=1, nlevels=4):
    """(bytes, flops) of one V-cycle over n fine rows with vb-byte values: the
    smoother's first forward sweep, its backward sweep (without the colour it
    turns at), the residual at the injected rows, the second smoother."""
    nb = fl = 0.0
    for level in range(nlevels):
        rows = n / 8.0 ** level
        sweeps = _FIRST / 27 + 7 / 8 + (0 if level == nlevels - 1 else 1 / 8 + 1 + 7 / 8)
        passes = 2 if level == nlevels - 1 else 4
        nb += rows * (sweeps * 27 * vb + nrhs * passes * 3 * vb)
        fl += rows * nrhs * sweeps * 54
    return nb, fl


def _iterations(case, n):
    """Iterations of a solve of n rows: given, or about what the tolerance takes
    (1e-9 on the reference matrix: they grow with the side; the diagonally
    dominant matrix of the differentiation problem: 17 for 1e-10)."""
    if case["tol"] == 0.0:
        return case["max_iter"]
    return 17 if case["kind"] == "adjoint" else round(0.63 * n ** (1 / 3)) + 1


def _solve(n, iters, vb=8, nrhs=1):
    vn, vf = _vcycle(n, vb, nrhs)
    nb = 27 * 8 * n + nrhs * n * (2 + 2 + 3 + 3 + 1) * 8 + vn  # SpMV, dots and vector updates, V-cycle
    return iters * nb, iters * (vf + nrhs * n * (54 + 12))


def work(case):
    kind = case["kind"]
    if kind == "vectors":
        n = case["n"]
        return dict(bytes=7 * 8.0 * n, flops=7.0 * n)
    if kind == "batch":
        rows = [d[0] * d[1] * d[2] for d in _batch_dims(case)]
        parts = [_solve(n, _iterations(case, n), 4) for n in rows]
        return dict(bytes=sum(p[0] for p in parts), flops=sum(p[1] for p in parts))
    n = float(case["nx"] * case["ny"] * case["nz"])
    if kind == "spmv":
        return dict(bytes=n * (27 * 8 + 16), flops=54 * n)
    if kind == "symgs":
        return dict(bytes=n * (2 * 27 * 8 + 6 * 8), flops=108 * n)
    if kind == "mg":
        nb, fl = _vcycle(n, 8)
        return dict(bytes=nb + 16 * n, flops=fl)
    if kind == "mg_f32":
        nb, fl = _vcycle(n, 4)
        return dict(bytes=nb + 24 * n, flops=fl)
    nrhs = case.get("nrhs", 1)
    nb, fl = _solve(n, _iterations(case, n), 4 if kind == "cg_mixed" else 8, nrhs)
    if kind == "adjoint":
        nb, fl = 2 * nb + 4 * 27 * 8 * n, 2 * fl + 27 * n
    return dict(bytes=nb, flops=fl)


# ---- the same results in plain torch, 64 bits ---------------------------------------

# The colours (parities of x, y, z as bits 0, 1, 2) in the order a forward sweep
# takes them; a backward sweep takes them in reverse from the last but one.
_SWEEP = (7, 6, 3, 5, 4, 1, 2, 0)


class _Grid:
    """One level: the 27-point matrix (26 and -1, or given values) on [nz, ny, nx] arrays."""

    def __init__(self, dims, values=None):
        self.nx, self.ny, self.nz = dims
        self.values = None if values is None else values.reshape(self.nz, self.ny, self.nx, 27)

    def pad(self, x):
        return torch.nn.functional.pad(x, (1, 1, 1, 1, 1, 1))

    def row_sums(self, xp, pz=0, py=0, px=0, step=1):
        """(A x) at points pz::step, ...; xp: x with a border of zeros."""
        nz, ny, nx = self.nz, self.ny, self.nx

        def cut(n, p, s):
            return slice(p + 1 + s, n + 1 + s, step)
        if self.values is None:
            t = sum(xp[:, :, cut(nx, px, s)] for s in (-1, 0, 1))
            t = sum(t[:, cut(ny, py, s)] for s in (-1, 0, 1))
            t = sum(t[cut(nz, pz, s)] for s in (-1, 0, 1))
            return 27.0 * xp[cut(nz, pz, 0), cut(ny, py, 0), cut(nx, px, 0)] - t
        a = self.values[pz::step, py::step, px::step]
        t = torch.zeros(a.shape[:3], device=xp.device, dtype=xp.dtype)
        for k, (sz, sy, sx) in enumerate(_directions()):
            t += a[..., k] * xp[cut(nz, pz, sz), cut(ny, py, sy), cut(nx, px, sx)]
        return t

    def matvec(self, x):
        return self.row_sums(self.pad(x))

    def symgs(self, r, x):
        xp = self.pad(x)
        inner = xp[1:-1, 1:-1, 1:-1]
        for c in _SWEEP + _SWEEP[-2::-1]:
            px, py, pz = c & 1, (c >> 1) & 1, (c >> 2) & 1
            mine = inner[pz::2, py::2, px::2]
            if mine.numel() == 0:
                continue
            d = 26.0 if self.values is None else self.values[pz::2, py::2, px::2, 13]
            mine += (r[pz::2, py::2, px::2] - self.row_sums(xp, pz, py, px, 2)) / d
        return inner.clone()


def _grids(dims, nlevels=4, values=None):
    return [_Grid(tuple(d >> i for d in dims), values if i == 0 else None) for i in range(nlevels)]


def _mg(grids, r):
    g = grids[0]
    x = g.symgs(r, torch.zeros_like(r))
    if len(grids) > 1:
        rc = r[::2, ::2, ::2] - g.row_sums(g.pad(x), step=2)
        x[::2, ::2, ::2] += _mg(grids[1:], rc)
        x = g.symgs(r, x)
    return x


def _pcg(grids, b, max_iter, tol, flexible=False):
    x = torch.zeros_like(b)
    r = b.clone()
    normr0 = normr = math.sqrt(float((r * r).sum()))
    k, p, rtz, zprev = 0, None, 0.0, None
    while k < max_iter and normr / normr0 > tol:
        z = _mg(grids, r)
        old, rtz = rtz, float((r * z).sum())
        if k == 0:
            p = z.clone()
        else:
            p = z + ((rtz - float((r * zprev).sum())) if flexible else rtz) / old * p
        zprev = z if flexible else None
        ap = grids[0].matvec(p)
        alpha = rtz / float((p * ap).sum())
        x += alpha * p
        r -= alpha * ap
        normr = math.sqrt(float((r * r).sum()))
        k += 1
    return x, k, normr, normr0


def exact(case, seed):
    kind = case["kind"]
    if kind == "vectors":
        n = case["n"]
        x, y = _uniform(seed, 0, n), _uniform(seed, 1, n)
        w = x - 0.75 * y
        return {"w": w, "dot": float((x * w).sum()), "residual": float((y - w).abs().max())}
    if kind == "batch":
        out = {"x": [], "iterations": None, "normr": None, "normr0": []}
        for i, d in enumerate(_batch_dims(case)):
            b = _uniform(seed, i, d[2], d[1], d[0])
            x, _, _, normr0 = _pcg(_grids(d), b, case["max_iter"], case["tol"], True)
            out["x"].append(x.reshape(-1))
            out["normr0"].append(normr0)
        out["normr0"] = np.array(out["normr0"])
        return out
    dims = _dims(case)
    shape = (dims[2], dims[1], dims[0])
    n = dims[0] * dims[1] * dims[2]
    if kind == "cg_multi":
        b = _uniform(seed, 0, case["nrhs"], n)
        got = [_pcg(_grids(dims), v.reshape(shape), case["max_iter"], case["tol"]) for v in b]
        return {"x": torch.stack([g[0].reshape(-1) for g in got]), "iterations": None,
                "normr": np.array([g[2] for g in got]), "normr0": np.array([g[3] for g in got])}
    b = _uniform(seed, 0, n).reshape(shape)
    if kind == "spmv":
        return {"y": _Grid(dims).matvec(b).reshape(-1)}
    if kind == "symgs":
        return {"x": _Grid(dims).symgs(b, _uniform(seed, 1, n).reshape(shape)).reshape(-1)}
    if kind in ("mg", "mg_f32"):
        return {"x": _mg(_grids(dims), b).reshape(-1)}
    if kind == "adjoint":
        v = _perturbed(dims, seed)
        grids = _grids(dims, 4, v)
        x = _pcg(grids, b, case["max_iter"], case["tol"])[0]
        lam = _pcg(grids, x - _uniform(seed, 1, n).reshape(shape), case["max_iter"], case["tol"])[0]
        xp = grids[0].pad(x)
        gv = torch.empty(*shape, 27, device=DEVICE, dtype=torch.float64)
        for k, (sz, sy, sx) in enumerate(_directions()):
            gv[..., k] = -lam * xp[1 + sz:1 + sz + shape[0], 1 + sy:1 + sy + shape[1], 1 + sx:1 + sx + shape[2]]
        return {"x": x.reshape(-1), "grad_values": gv.reshape(n, 27), "grad_b": lam.reshape(-1)}
    x, _, normr, normr0 = _pcg(_grids(dims), b, case["max_iter"], case["tol"], kind == "cg_mixed")
    return {"x": x.reshape(-1), "iterations": None, "normr": normr if case["tol"] == 0.0 else None, "normr0": normr0}
