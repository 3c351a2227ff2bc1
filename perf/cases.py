"""Timed workloads of libab2 through its Python entry points (alien_b200/abi.py).

    listed()             the workloads, by name
    draw(rng)            one more workload of the same ranges
    prepare(case, seed)  inputs, plans and handles a program holds before the call
    run(state)           one pass; returns what the pass computes
    work(case)           bytes and operations one pass cannot do without
    exact(case, seed)    the same results in 64 bits, by torch alone, where they exist

Systems: 3-D 7-point (2-D 5-point with nz = 1) matrices in lexicographic
order, assembled here with torch from the seed -- constant-coefficient
Poisson, heterogeneous diffusion (log10 k a smoothed Gaussian random field,
harmonic-mean faces, Dirichlet boundaries) and convection-diffusion (unit
diffusion, first-order upwind, a divergence-free velocity from 8 random
Fourier modes, cell Peclet number up to 10) -- and ragged matrices with
scattered columns.  The right-hand side of a solve is b = A x_true with
x_true uniform in [-1, 1].
"""
from __future__ import annotations

import math
from pathlib import Path

import numpy as np
import torch

from alien_b200 import abi

WEIGHTS = Path(abi.__file__).resolve().parent / "gnn_weights.npy"
GRID_FORMATS = abi.FMT_CSR | abi.FMT_ELL | abi.FMT_STENCIL


# ---------------------------------------------------------------------------- cases
def listed() -> list[dict]:
    return [
        # a small system solved again and again with one solver: every launch counts
        dict(name="cg_diag_poisson_32", kind="cg_diag", field="poisson", nx=32, ny=32, nz=32),
        # a mid-size box with odd sides, solver kept: the matrix sits in L2
        dict(name="cg_diag_diffusion_97x61x83", kind="cg_diag", field="diffusion", nx=97, ny=61, nz=83),
        # the drop-in path at scale: ILU(0) set-up and solve per matrix
        dict(name="cg_ilu0_diffusion_192", kind="cg_ilu0", field="diffusion", nx=192, ny=192, nz=192),
        # the same path on a box smaller than L2 with ragged sides
        dict(name="cg_ilu0_diffusion_70x90x50", kind="cg_ilu0", field="diffusion", nx=70, ny=90, nz=50),
        # Chebyshev(3), Lanczos bounds, set-up included
        dict(name="cg_cheb_diffusion_160x152x144", kind="cg_cheb", field="diffusion", nx=160, ny=152, nz=144),
        # FP32 inner solves in FP64 refinement, nonsymmetric: BiCGStab + ILU(0) to 1e-10
        dict(name="mixed_bicg_ilu0_convdiff_128", kind="mixed_ilu0", field="convdiff", nx=128, ny=128, nz=128),
        # FP32 inner Jacobi-CG at scale
        dict(name="mixed_diag_diffusion_192", kind="mixed_diag", field="diffusion", nx=192, ny=192, nz=192),
        # a matrix that is no 3-D grid: BiCGStab + ILU(0) by wavefronts
        dict(name="bicg_ilu0_convdiff2d_181x140", kind="bicg_ilu0", field="convdiff", nx=181, ny=140, nz=1),
        # many independent systems of uneven sizes in one launch
        dict(name="batch_96", kind="batch", field="diffusion", nsys=96, rows_min=2000, rows_max=200000),
        # the learned preconditioner inside flexible CG, ILU(0) after failed steps
        dict(name="fcg_gnn_diffusion_128x120x112", kind="fcg", field="diffusion", nx=128, ny=120, nz=112),
        # training of that preconditioner: loss and gradient of one (residual, error) pair
        dict(name="gnn_grad_diffusion_64", kind="gnn_grad", field="diffusion", nx=64, ny=64, nz=64),
        # Alien's templates over the algebra: one CG iteration in single calls, ragged rows
        dict(name="algebra_ragged_20011", kind="algebra", field="ragged", n=20011, row_min=4, row_max=12),
    ]


#: (log-uniform side range, field) of the drawn grid cases of each kind
_RANGES = {
    "cg_diag": (12, 128, ("poisson", "diffusion")),
    "cg_ilu0": (16, 128, ("diffusion",)),
    "cg_cheb": (20, 128, ("diffusion",)),
    "mixed_ilu0": (24, 112, ("convdiff",)),
    "mixed_diag": (24, 160, ("diffusion",)),
    "bicg_ilu0": (24, 160, ("convdiff",)),
    "fcg": (24, 96, ("diffusion",)),
    "gnn_grad": (16, 64, ("diffusion",)),
}


def _log_int(rng, lo: float, hi: float) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["cg_diag", "cg_diag", "cg_ilu0", "cg_ilu0", "cg_cheb", "mixed_ilu0", "mixed_diag", "bicg_ilu0",
                       "batch", "fcg", "gnn_grad", "algebra", "algebra"])
    if kind == "algebra":
        return dict(kind=kind, field="ragged", n=_log_int(rng, 1500, 2_500_000), row_min=rng.randint(2, 6),
                    row_max=rng.randint(8, 24))
    if kind == "batch":
        return dict(kind=kind, field="diffusion", nsys=rng.randint(24, 96), rows_min=2000,
                    rows_max=_log_int(rng, 20000, 200000))
    lo, hi, fields = _RANGES[kind]
    side = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    dims = [max(8, min(hi, int(round(side * rng.uniform(0.75, 1.3))))) for _ in range(3)]
    if kind == "bicg_ilu0":
        dims[2] = 1
    return dict(kind=kind, field=rng.choice(fields), nx=dims[0], ny=dims[1], nz=dims[2])


# ---------------------------------------------------------------------------- inputs
def _dev() -> str:
    return "cuda" if torch.cuda.is_available() else "cpu"


def _gen(seed: int, stream: int) -> torch.Generator:
    return torch.Generator(_dev()).manual_seed(1000003 * int(seed) + stream)


def _smoothed_field(shape, sigma: float, length: float, g: torch.Generator) -> torch.Tensor:
    """Gaussian random field on `shape`, smoothed over `length` cells, mean 0, std sigma."""
    f = torch.randn(shape, generator=g, device=g.device, dtype=torch.float64)
    spec = torch.fft.rfftn(f)
    for ax, m in enumerate(shape):
        k = torch.fft.rfftfreq(m, device=g.device) if ax == len(shape) - 1 else torch.fft.fftfreq(m, device=g.device)
        damp = torch.exp(-2.0 * (math.pi * length * k.double()) ** 2)
        spec = spec * damp.reshape([-1 if a == ax else 1 for a in range(len(shape))])
    f = torch.fft.irfftn(spec, s=list(shape))
    f = f - f.mean()
    return f * (sigma / f.std())


def _row_sums(row_ptr, entries):
    """Sums of each row's entries, slot by slot: the same bits on every run."""
    begin, end = row_ptr[:-1].long(), row_ptr[1:].long()
    sums = entries.new_zeros(begin.numel())
    for j in range(int((end - begin).max())):
        at = begin + j
        sums = sums + torch.where(at < end, entries[at.clamp(max=entries.numel() - 1)], 0.0)
    return sums


class _System:
    """A CSR system on the device: row_ptr, cols (int32), vals, x_true, b."""

    def __init__(self, row_ptr, cols, vals, g):
        self.row_ptr, self.cols, self.vals = row_ptr, cols, vals
        self.n = row_ptr.numel() - 1
        self.x_true = torch.rand(self.n, generator=g, device=g.device, dtype=torch.float64) * 2 - 1
        self.b = self.mult(self.x_true)

    def rows(self):
        return torch.repeat_interleave(torch.arange(self.n, device=self.cols.device),
                                       (self.row_ptr[1:] - self.row_ptr[:-1]).long())

    def mult(self, x):
        return _row_sums(self.row_ptr, self.vals * x[self.cols.long()])

    def matrix(self, ctx, formats):
        return ctx.matrix(self.row_ptr.cpu().numpy(), self.cols.cpu().numpy(), self.vals.cpu().numpy(), formats)


def _grid_csr(nz, ny, nx, lower_upper, diag):
    """CSR of a grid matrix; lower_upper: per axis (z, y, x) the off-diagonal
    value of every cell towards its -1 and +1 neighbour (as (nz, ny, nx) arrays)."""
    dev = diag.device
    idx = torch.arange(nz * ny * nx, device=dev).reshape(nz, ny, nx)
    strides = (ny * nx, nx, 1)
    cols, vals, keep = [], [], []
    for sign, axes in ((-1, (0, 1, 2)), (0, (None,)), (1, (2, 1, 0))):  # ascending columns
        for ax in axes:
            if ax is None:
                cols.append(idx)
                vals.append(diag)
                keep.append(torch.ones_like(idx, dtype=torch.bool))
                continue
            if diag.shape[ax] == 1:
                continue
            c = torch.arange(diag.shape[ax], device=dev).reshape([-1 if a == ax else 1 for a in range(3)])
            inside = (c > 0) if sign < 0 else (c < diag.shape[ax] - 1)
            cols.append(idx + sign * strides[ax])
            vals.append(lower_upper[ax][0 if sign < 0 else 1])
            keep.append(inside.expand(nz, ny, nx))
    cols, vals, keep = (torch.stack([t.reshape(-1) for t in v], 1) for v in (cols, vals, keep))
    row_ptr = torch.zeros(idx.numel() + 1, dtype=torch.int64, device=dev)
    row_ptr[1:] = keep.sum(1).cumsum(0)
    return row_ptr.int(), cols[keep].int(), vals[keep]


def _diffusion(nx, ny, nz, sigma, length, g):
    k = 10.0 ** _smoothed_field((nz, ny, nx), sigma, length, g)
    diag = torch.zeros_like(k)
    lu = []
    for ax in range(3):
        if k.shape[ax] == 1:
            lu.append(None)
            continue
        m = k.shape[ax]
        a, b = k.narrow(ax, 0, m - 1), k.narrow(ax, 1, m - 1)
        t = 2.0 * a * b / (a + b)
        lo, up = torch.zeros_like(k), torch.zeros_like(k)
        lo.narrow(ax, 1, m - 1).copy_(-t)
        up.narrow(ax, 0, m - 1).copy_(-t)
        face_lo, face_up = -lo, -up
        face_lo.narrow(ax, 0, 1).copy_(2.0 * k.narrow(ax, 0, 1))  # Dirichlet faces at half a cell
        face_up.narrow(ax, m - 1, 1).copy_(2.0 * k.narrow(ax, m - 1, 1))
        diag += face_lo
        diag += face_up
        lu.append((lo, up))
    return _grid_csr(nz, ny, nx, lu, diag)


def _poisson(nx, ny, nz, g):
    one = torch.ones((nz, ny, nx), dtype=torch.float64, device=g.device)
    return _grid_csr(nz, ny, nx, [(-one, -one)] * 3, one * (6.0 if nz > 1 else 4.0))


def _convdiff(nx, ny, nz, peclet, modes, g):
    """Upwind convection-diffusion; face fluxes are the circulation of a
    vector potential on the cell edges, so every cell's net flux is zero."""
    dev, span = g.device, 2.0 * math.pi / max(nx, ny, nz)
    kv = torch.randint(-3, 4, (modes, 3), generator=g, device=dev).double()
    kv[(kv == 0).all(1), 0] = 1.0
    amp = torch.randn((modes, 3), generator=g, device=dev, dtype=torch.float64) / kv.norm(dim=1, keepdim=True)
    ph = 2.0 * math.pi * torch.rand((modes, 3), generator=g, device=dev, dtype=torch.float64)

    def psi(c, x0, y0, z0):
        ax = [torch.arange(m + 1, device=dev).double() + o for m, o in ((nz, z0), (ny, y0), (nx, x0))]
        s = torch.zeros((nz + 1, ny + 1, nx + 1), dtype=torch.float64, device=dev)
        for m in range(modes):
            arg = (kv[m, 2] * ax[0])[:, None, None] + (kv[m, 1] * ax[1])[None, :, None] + (kv[m, 0] * ax[2])[None, None]
            s += amp[m, c] * torch.sin(span * arg + ph[m, c])
        return s

    ez = psi(2, 0, 0, 0.5 if nz > 1 else 0.0)
    if nz > 1:
        ex, ey = psi(0, 0.5, 0, 0), psi(1, 0, 0.5, 0)
    else:
        ex = ey = torch.zeros_like(ez)
    fx = (ey[:-1, :-1, :] + ez[:-1, 1:, :] - ey[1:, :-1, :] - ez[:-1, :-1, :])
    fy = (ez[:-1, :, :-1] + ex[1:, :, :-1] - ez[:-1, :, 1:] - ex[:-1, :, :-1])
    fz = (ex[:, :-1, :-1] + ey[:, :-1, 1:] - ex[:, 1:, :-1] - ey[:, :-1, :-1])
    scale = peclet / max(float(f.abs().max()) for f in (fx, fy, fz))
    diag = torch.zeros((nz, ny, nx), dtype=torch.float64, device=dev)
    lu = []
    for ax, f in enumerate((fz, fy, fx)):
        m = diag.shape[ax]
        if m == 1:
            lu.append(None)
            continue
        pair = []
        for out, edge in ((-scale * f.narrow(ax, 0, m), 0), (scale * f.narrow(ax, 1, m), m - 1)):
            pair.append(-1.0 + out.clamp(max=0.0))
            d = 1.0 + out.clamp(min=0.0)
            d.narrow(ax, edge, 1).add_(1.0)
            diag += d
        lu.append(tuple(pair))
    return _grid_csr(nz, ny, nx, lu, diag)


def _ragged(n, row_min, row_max, g):
    """Rows of row_min..row_max entries, columns scattered over a window of
    about n^(2/3) rows around the diagonal; diagonally dominant."""
    dev, span = g.device, max(row_max, int(round(n ** (2.0 / 3.0))))
    row = torch.arange(n, device=dev)
    length = torch.randint(row_min, row_max + 1, (n,), generator=g, device=dev)
    off = torch.randint(-span, span + 1, (n, row_max), generator=g, device=dev)
    off[:, 0] = 0
    keep = torch.arange(row_max, device=dev)[None] < length[:, None]
    key = (row[:, None] * n + (row[:, None] + off).clamp(0, n - 1))[keep].unique()
    rows, cols = key // n, key % n
    vals = -torch.rand(key.numel(), generator=g, device=dev, dtype=torch.float64)
    row_ptr = torch.zeros(n + 1, dtype=torch.int64, device=dev)
    row_ptr[1:] = torch.bincount(rows, minlength=n).cumsum(0)
    vals[rows == cols] = _row_sums(row_ptr, vals.abs()) + 0.1  # one diagonal entry a row, in row order
    return row_ptr.int(), cols.int(), vals


def _grid_system(case, seed) -> _System:
    g = _gen(seed, 1)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    if case["field"] == "poisson":
        csr = _poisson(nx, ny, nz, g)
    elif case["field"] == "convdiff":
        csr = _convdiff(nx, ny, nz, 10.0, 8, g)
    elif case["kind"] in ("fcg", "gnn_grad"):  # the learned form's fields: std 1.5, smoothing drawn in [2, 8] cells
        csr = _diffusion(nx, ny, nz, 1.5, 2.0 + 6.0 * float(torch.rand(1, generator=g, device=g.device)), g)
    else:
        csr = _diffusion(nx, ny, nz, 1.0, 4.0, g)
    return _System(*csr, g)


def _batch_dims(case) -> list[tuple]:
    """Half 2-D squares, half 3-D cubes, rows log-uniform over the range (the
    same shapes for every seed; the coefficients are the seed's)."""
    dims, m = [], case["nsys"]
    for s in range(m):
        rows = math.exp(math.log(case["rows_min"]) + (s * 0.6180339887 % 1.0) * math.log(case["rows_max"] / case["rows_min"]))
        side = max(2, int(round(rows ** (1 / 2 if s % 2 else 1 / 3))))
        dims.append((side, side, 1) if s % 2 else (side, side, side))
    return dims


def _batch_system(case, seed):
    g = _gen(seed, 2)
    row_ptr, cols, vals, offs, e = [torch.zeros(1, dtype=torch.int32, device=g.device)], [], [], [0], 0
    for nx, ny, nz in _batch_dims(case):
        rp, ci, v = _diffusion(nx, ny, nz, 1.0, 2.0, g)
        row_ptr.append(rp[1:] + e)
        cols.append(ci + offs[-1])
        vals.append(v)
        offs.append(offs[-1] + rp.numel() - 1)
        e += v.numel()
    return _System(torch.cat(row_ptr), torch.cat(cols), torch.cat(vals), g), np.asarray(offs, dtype=np.int32)


def _pair(case, system, seed):
    """A (residual, error) pair of the training distribution: a smooth error and r = A e."""
    e = _smoothed_field((case["nz"], case["ny"], case["nx"]), 1.0, 1.5, _gen(seed, 3)).reshape(-1)
    return system.mult(e), e


def _algebra_vectors(n, seed):
    g = _gen(seed, 4)
    return [torch.rand(n, generator=g, device=g.device, dtype=torch.float64) * 2 - 1 for _ in range(4)]


# ---------------------------------------------------------------------------- one pass
class _DeviceArray:
    """A vector's device memory for torch (shares it and keeps the vector alive)."""

    def __init__(self, vector):
        self.vector = vector
        self.__cuda_array_interface__ = {"shape": (vector.n,), "typestr": "<f8", "data": (vector.device_ptr, False),
                                         "version": 3, "strides": None}


def _tensor(vector):
    return torch.as_tensor(_DeviceArray(vector), device="cuda")


SOLVER_OPTIONS = {
    "cg_diag": dict(solver="cg", precond="diag", tol=1e-8, max_iter=4000),
    "cg_ilu0": dict(solver="cg", precond="ilu0", tol=1e-8, max_iter=2000),
    "cg_cheb": dict(solver="cg", precond="cheb", tol=1e-8, max_iter=2000, cheb_saad=True, cheb_lanczos=True,
                    poly_order=3, poly_factor_max_iter=20),
    "bicg_ilu0": dict(solver="bicgs", precond="ilu0", tol=1e-8, max_iter=2000),
    "mixed_ilu0": dict(solver="bicgs", precond="ilu0", tol=1e-10),
    "mixed_diag": dict(solver="cg", precond="diag", tol=1e-8, inner_max_iter=4000),
}


def prepare(case, seed):
    kind = case["kind"]
    ctx = abi.Context(0)
    s = {"kind": kind, "ctx": ctx}
    if kind == "algebra":
        system = _System(*_ragged(case["n"], case["row_min"], case["row_max"], _gen(seed, 1)), _gen(seed, 5))
        s["A"] = system.matrix(ctx, abi.FMT_CSR | abi.FMT_ELL)
        for name, v in zip("prxd", _algebra_vectors(system.n, seed)):
            s[name + "0"] = ctx.vector(v.cpu().numpy())
            s[name] = ctx.vector(system.n)
        s["q"], s["z"] = ctx.vector(system.n), ctx.vector(system.n)
        ctx.computeInvDiag(s["A"], s["d"])
        return s
    if kind == "batch":
        system, offs = _batch_system(case, seed)
        s["A"] = system.matrix(ctx, abi.FMT_CSR | abi.FMT_ELL | abi.FMT_F32)
        s["plan"] = abi.Batch(ctx, s["A"], offs, tol=1e-8, cluster_size=8, threads=512, spmv_variant=abi.SPMV_ELL,
                              ell_slice=64, lanes_per_row=1)
    else:
        system = _grid_system(case, seed)
        formats = abi.FMT_CSR | abi.FMT_ELL if kind == "bicg_ilu0" else GRID_FORMATS
        s["A"] = system.matrix(ctx, formats | (abi.FMT_F32 if kind.startswith("mixed") else 0))
    if kind == "gnn_grad":
        r, e = _pair(case, system, seed)
        s["r"], s["e"] = ctx.vector(r.cpu().numpy()), ctx.vector(e.cpu().numpy())
    else:
        s["b"], s["x"] = ctx.vector(system.b.cpu().numpy()), ctx.vector(system.n)
    if kind in ("fcg", "gnn_grad"):
        s["net"] = abi.Gnn(ctx, np.load(WEIGHTS))
        s["net"].bind(s["A"])
    if kind == "cg_diag":
        s["solver"] = abi.Solver(ctx, s["A"], **SOLVER_OPTIONS[kind])
    return s


def run(s):
    kind, ctx = s["kind"], s["ctx"]
    if kind == "algebra":
        return _cg_step_in_calls(s)
    if kind == "gnn_grad":
        loss, grad = s["net"].loss_grad(s["r"], s["e"])
        return {"loss": loss, "grad": grad}
    A, b, x = s["A"], s["b"], s["x"]
    ctx.assign(x, 0.0)
    if kind == "cg_diag":
        s["solver"].solve(b, x)
    elif kind == "batch":
        s["plan"].solve(b, x)
    elif kind == "fcg":
        pc = abi.Precond(ctx, A, "ilu0")
        abi.fcg_solve(ctx, A, b, x, gnn=s["net"], fallback=pc, tol=1e-8, max_iter=3000, fallback_ratio=1.0)
        pc.close()
    else:
        form = abi.Mixed if kind.startswith("mixed") else abi.Solver
        solver = form(ctx, A, **SOLVER_OPTIONS[kind])
        solver.solve(b, x)
        solver.close()
    return {"x": _tensor(x)}


def _cg_step_in_calls(s):
    """The calls of one Jacobi-CG iteration as Alien's templates make them."""
    ctx, A, p, q, r, x, z, d = (s[k] for k in ("ctx", "A", "p", "q", "r", "x", "z", "d"))
    for k in "prx":
        ctx.copy(s[k + "0"], s[k])
    ctx.pointwiseMult(d, r, z)
    rho = ctx.dot(r, z)
    ctx.mult(A, p, q)
    alpha = rho / ctx.dot(q, p)
    ctx.axpy(alpha, p, x)
    ctx.axpy(-alpha, q, r)
    rr = ctx.dot(r, r)
    ctx.pointwiseMult(d, r, z)
    rho1 = ctx.dot(r, z)
    ctx.scal(rho1 / rho, p)
    ctx.axpy(1.0, z, p)
    return {"x": _tensor(x), "r": _tensor(r), "p": _tensor(p), "rr": rr, "norm": ctx.norm2(r)}


# ---------------------------------------------------------------------------- bounds and results
def work(case):
    """A solve reads the matrix (in the path's compact form) and b once and
    writes x once per Krylov iteration it cannot do without; the iteration
    count is the method's own, taken here as a fixed multiple of the longest
    side, so the figures compare sizes, not convergence."""
    kind = case["kind"]
    if kind == "algebra":
        nnz = case["n"] * (case["row_min"] + case["row_max"]) / 2
        return {"bytes": 12 * nnz + 4 * case["n"] + 8 * 33 * case["n"], "flops": 2 * nnz + 16 * case["n"]}
    dims = _batch_dims(case) if kind == "batch" else [(case["nx"], case["ny"], case["nz"])]
    total = {"bytes": 0.0, "flops": 0.0}
    for nx, ny, nz in dims:
        n, side = float(nx * ny * nz), max(nx, ny, nz)
        if kind == "gnn_grad":  # activations of five layers in BF16 out and back, their gradients in FP32
            total["bytes"] += n * (5 * 64 * 2 * 2 + 5 * 64 * 4 * 2)
            total["flops"] += 3 * n * 4 * (2 * 64 * 128 + 2 * 6 * 64)
            continue
        # per iteration and row: four FP64 bands and the vectors of a CG step (a factor's seven bands more for ILU(0)),
        # half of it in FP32
        per_row = {"cg_diag": 96, "cg_ilu0": 176, "cg_cheb": 300, "mixed_ilu0": 200, "mixed_diag": 56,
                   "bicg_ilu0": 500, "batch": 100, "fcg": 1200}[kind]
        its = {"cg_diag": 3.3, "cg_ilu0": 1.4, "cg_cheb": 1.5, "mixed_ilu0": 0.9, "mixed_diag": 3.5, "bicg_ilu0": 0.6,
               "batch": 8.0, "fcg": 1.3}[kind]
        total["bytes"] += n * per_row * its * side
        total["flops"] += n * its * side * (4 * 2 * 64 * 128 if kind == "fcg" else 40)
    return total


def exact(case, seed):
    kind = case["kind"]
    if kind == "algebra":
        system = _System(*_ragged(case["n"], case["row_min"], case["row_max"], _gen(seed, 1)), _gen(seed, 5))
        p, r, x, _ = _algebra_vectors(system.n, seed)
        d = 1.0 / system.vals[system.cols.long() == system.rows()]
        rho, q = r @ (d * r), system.mult(p)
        alpha = rho / (q @ p)
        x, r = x + alpha * p, r - alpha * q
        rr, rho1 = r @ r, r @ (d * r)
        return {"x": x, "r": r, "p": d * r + (rho1 / rho) * p, "rr": float(rr), "norm": float(rr.sqrt())}
    if kind == "gnn_grad":
        system = _grid_system(case, seed)
        return _network_loss_grad(system, *_pair(case, system, seed))
    system = _batch_system(case, seed)[0] if kind == "batch" else _grid_system(case, seed)
    return {"x": system.x_true}


def _network_loss_grad(system, r, e):
    """Loss and gradient of the message-passing network in FP64, by autograd
    over the six neighbour directions of the grid graph."""
    w = torch.from_numpy(np.load(WEIGHTS).astype(np.float64)).to(r.device).requires_grad_(True)
    sizes = [128, 64] + [64 * 128] * 4 + [64] * 4 + [4, 4, 64, 1, 1]
    W0, b0, *rest = torch.split(w, sizes)
    W, b, (u, c, wd, bd, ws) = rest[:4], rest[4:8], rest[8:]
    rows = system.rows()
    off = rows != system.cols.long()
    rows, cols, vals = rows[off], system.cols[off].long(), system.vals[off]
    diag = system.vals[~off]
    feat = vals.abs().log() - 0.5 * (diag[rows].log() + diag[cols].log())
    sd = diag.sqrt()
    t = r / sd
    scale = t.square().mean().sqrt()
    x0 = torch.stack([t / scale, diag.log() / 10.0], 1)
    h = torch.relu(x0 @ W0.reshape(64, 2).T + b0)
    for layer in range(4):
        gate = torch.sigmoid(u[layer] * feat + c[layer])
        m = torch.zeros_like(h).index_add(0, rows, gate[:, None] * h[cols])
        h = torch.relu(torch.cat([h, m], 1) @ W[layer].reshape(64, 128).T + b[layer])
    z = scale * (h @ wd + bd + ws * x0[:, 0]) / sd
    err = z - e
    loss = (err @ system.mult(err)) / (e @ system.mult(e))
    loss.backward()
    return {"loss": float(loss.detach()), "grad": w.grad.float()}
