"""Measured cases: the calls a user of this AMG library makes, on device
vectors, over the range of sizes and options they are made with.

Kinds of pass (each through the package's public functions):
  cycle    amg_cycle: one V or W cycle on the caller's vectors, the
           preconditioner application of a host Krylov method
  solve    amg_solve: the stationary AMG iteration
  pcg      AMG-preconditioned CG to 1e-8, FP64 or FP32 cycle
  fgmres   flexible GMRES(30) to 1e-8 on a nonsymmetric operator
  block    pcg_multi: one matrix, k right-hand sides
  batch    pcg_batched: many independent systems at once
  resetup  new coefficients on the device (Galerkin products, smoothers,
           coarsest factors), then one cycle with the refreshed hierarchy
  adjoint  amg_solve_diff forward and backward: resetup, solve, transposed
           solve, gradients of the matrix values and the right-hand side

A program keeps its hierarchy and calls with new right-hand sides or new
coefficients, so the matrix of a case is fixed by the case and the seed
makes the vectors and coefficients; the hierarchy of the case in hand is
kept (one at a time) and shared by the states prepared for it.
"""

import math
import pathlib
import sys

import numpy as np
import torch

sys.path.insert(0, str(pathlib.Path(__file__).resolve().parent.parent / "draugr.jl_b200"))
import draugr  # noqa: E402
from draugr import problems  # noqa: E402

F64 = torch.float64
SMOOTHERS = {"jacobi": draugr.JacobiSmootherType, "l1_jacobi": draugr.L1JacobiSmootherType,
             "spai0": draugr.SPAI0SmootherType, "chebyshev": draugr.ChebyshevSmootherType,
             "l1_colored_gs": draugr.L1ColoredGaussSeidelType, "colored_gs": draugr.ColoredGaussSeidelType}
JACOBI_TYPE = ("jacobi", "l1_jacobi", "spai0")
CHEB_DEGREE = 3


def _case(name, kind, problem, n, config="hypre", smoother="l1_jacobi", precision="fp64", cycle="V", k=1):
    return {"name": name, "kind": kind, "problem": problem, "n": n, "config": config, "smoother": smoother,
            "precision": precision, "cycle": cycle, "k": k}


def listed():
    return [
        # a small system inside a host's own Krylov loop: latency and launches
        _case("cycle_2d_47", "cycle", "poisson2d", 47, "default", "l1_colored_gs"),
        # an ordinary ragged 3-D system preconditioned from outside
        _case("cycle_3d_41", "cycle", "het3d", 41),
        # the preconditioner application at the headline size
        _case("cycle_3d_128", "cycle", "het3d", 128),
        # the headline solve: heterogeneous diffusion, FP64 throughout
        _case("pcg_3d_128", "pcg", "het3d", 128),
        # an ordinary odd-sized solve with the FP32 cycle
        _case("pcg_3d_101_mixed", "pcg", "het3d", 101, precision="mixed"),
        # the package's default configuration (HMIS, l1 colored Gauss-Seidel)
        _case("pcg_3d_64_default", "pcg", "het3d", 64, "default", "l1_colored_gs"),
        # the stationary solver on the reference's 2-D model problem
        _case("solve_2d_256", "solve", "poisson2d", 256, "aggregation", "jacobi"),
        # a convection-diffusion system
        _case("fgmres_2d_300_mixed", "fgmres", "convdiff2d", 300, precision="mixed"),
        # many right-hand sides of one matrix
        _case("block_3d_96_k32", "block", "het3d", 96, precision="mixed", k=32),
        # many uneven systems
        _case("batch_64_mixed", "batch", "poisson3d", 64, precision="mixed", k=64),
        # a coefficient update of a time-stepping or optimisation loop
        _case("resetup_27pt_96", "resetup", "fe27", 96),
        # a gradient through the solve
        _case("adjoint_2d_256", "adjoint", "convdiff2d", 256),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["cycle", "cycle", "pcg", "pcg", "solve", "fgmres", "block", "batch", "resetup", "adjoint"])
    precision = rng.choice(["fp64", "mixed"])
    c = None
    if kind == "cycle":
        three = rng.random() < 0.7
        config, smoother = rng.choice([("hypre", "l1_jacobi"), ("hypre", "l1_jacobi"), ("hypre", "chebyshev"),
                                       ("hypre", "spai0"), ("default", "l1_colored_gs"),
                                       ("aggregation", "colored_gs")])
        c = _case("", kind, "het3d" if three else "poisson2d", size(12, 112) if three else size(24, 700), config,
                  smoother, cycle=rng.choice(["V", "V", "V", "W"]))
    elif kind == "pcg":
        config, smoother = rng.choice([("hypre", "l1_jacobi"), ("hypre", "l1_jacobi"), ("hypre", "spai0"),
                                       ("default", "l1_colored_gs")])
        c = _case("", kind, "het3d", size(12, 64 if config == "default" else 112), config, smoother, precision)
    elif kind == "solve":
        c = _case("", kind, "poisson2d", size(24, 400), "aggregation", rng.choice(["jacobi", "l1_jacobi"]))
    elif kind == "fgmres":
        c = _case("", kind, "convdiff2d", size(24, 400), precision=precision)
    elif kind == "block":
        c = _case("", kind, "het3d", size(16, 80), precision=precision, k=rng.choice([1, 3, 5, 8, 12, 16, 20, 32]))
    elif kind == "batch":
        c = _case("", kind, "poisson3d", size(20, 56), precision=precision, k=size(3, 48))
    elif kind == "resetup":
        c = _case("", kind, "fe27", size(14, 80))
    else:
        two = rng.random() < 0.6
        c = _case("", kind, "convdiff2d" if two else "het3d", size(24, 300) if two else size(10, 48),
                  precision=precision)
    del c["name"]
    return c


# ------------------------------------------------------------ matrices

def _config(case):
    smoother = SMOOTHERS[case["smoother"]]()
    if case["config"] == "hypre":
        return draugr.hypre_default_config(agg_trunc_factor=0.2, smoother=smoother, cycle_type=case["cycle"], seed=3)
    if case["config"] == "default":
        return draugr.AMGConfig(smoother=smoother, cycle_type=case["cycle"], seed=3)
    return draugr.AMGConfig(coarsening=draugr.AggregationCoarsening(0.25), smoother=smoother,
                            cycle_type=case["cycle"], seed=3)


def _fe27(m, kappa):
    """(rowptr, columns, values) of the 27-point Q1 operator on m^3 nodes
    with one coefficient per element (kappa: (m+1)^3 on the GPU), assembled
    on the GPU."""
    eps = (1.0, 1.0, 1e-3)
    ax = torch.arange(m, device="cuda")
    z, y, x = torch.meshgrid(ax, ax, ax, indexing="ij")
    vals, valid, offs = [], [], []
    for dz in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                acc = torch.zeros((m, m, m), dtype=F64, device="cuda")
                for sz in (0, 1):
                    for sy in (0, 1):
                        for sx in (0, 1):
                            lz, ly, lx = 1 - sz, 1 - sy, 1 - sx
                            mz, my, mx = lz + dz, ly + dy, lx + dx
                            if 0 <= mz <= 1 and 0 <= my <= 1 and 0 <= mx <= 1:
                                w = float(problems.q1_element_entry(lx, ly, lz, mx, my, mz, eps))
                                acc += w * kappa[sz:sz + m, sy:sy + m, sx:sx + m]
                vals.append(acc.reshape(-1))
                valid.append(((x + dx >= 0) & (x + dx < m) & (y + dy >= 0) & (y + dy < m) & (z + dz >= 0)
                              & (z + dz < m)).reshape(-1))
                offs.append(dz * m * m + dy * m + dx)
    mask = torch.stack(valid, 1)
    cols = torch.arange(m ** 3, device="cuda")[:, None] + torch.tensor(offs, device="cuda")[None, :]
    rp = torch.zeros(m ** 3 + 1, dtype=torch.int64, device="cuda")
    rp[1:] = torch.cumsum(mask.sum(1), 0)
    return rp, cols[mask], torch.stack(vals, 1)[mask]


def _matrix(case):
    """(n, rowptr, columns, values) on the host, the same for every seed."""
    m = case["n"]
    if case["problem"] == "fe27":
        rp, ci, v = _fe27(m, torch.ones((m + 1,) * 3, dtype=F64, device="cuda"))
        return m ** 3, rp.cpu().numpy(), ci.cpu().numpy(), v.cpu().numpy()
    if case["problem"] == "het3d":
        A = problems.heterogeneous_diffusion_3d(m, seed=11)
    elif case["problem"] == "poisson2d":
        A = problems.poisson2d(m, m + 1)
    elif case["problem"] == "poisson3d":
        A = problems.poisson3d(m)
    else:
        kappa = np.exp(0.5 * np.random.default_rng(11).standard_normal((m, m)))
        A, _ = problems.convection_diffusion_2d(kappa, 50.0, seed=5)
    return A.shape[0], A.indptr, A.indices, A.data


def _sides(case):
    """Grid sides of a batch's systems: uneven, n the largest."""
    return np.random.default_rng(7).integers(max(8, case["n"] // 4), case["n"] + 1, size=case["k"])


class _Plan:
    """What a program keeps for a case: the matrix, its hierarchy, a stream."""

    def __init__(self, case):
        self.config = _config(case)
        self.stream = torch.cuda.Stream()
        if case["kind"] == "batch":
            mats = [problems.poisson3d(int(s)) for s in _sides(case)]
            self.parts = [draugr.amg_setup(A, self.config) for A in mats]
            self.h = draugr.batch_setup(self.parts, self.config)
            self.A = None
            self.mats = mats
            self.n = self.h.n
        else:
            self.A = _matrix(case)
            self.n = self.A[0]
            self.h = draugr.amg_setup(self.A, self.config)
        self.h.set_stream(self.stream)


_kept = {}


def _plan(case):
    key = repr(sorted((a, b) for a, b in case.items() if a != "name"))
    if key not in _kept:
        _kept.clear()
        _kept[key] = _Plan(case)
    return _kept[key]


# ------------------------------------------------------------ passes

def prepare(case, seed):
    plan = _plan(case)
    n, kind = plan.n, case["kind"]
    g = torch.Generator(device="cuda").manual_seed(int(seed))

    def uniform(*shape):
        return 2.0 * torch.rand(shape, dtype=F64, device="cuda", generator=g) - 1.0

    s = {"case": case, "plan": plan, "x": torch.empty(n, dtype=F64, device="cuda")}
    if kind == "block":
        s["b"] = uniform(n, case["k"])
        s["x"] = torch.empty_like(s["b"])
    else:
        s["b"] = uniform(n)
    if kind in ("cycle", "resetup"):
        s["x0"] = uniform(n)
    if kind == "resetup":
        m = case["n"]
        kappa = torch.exp(0.5 * torch.randn((m + 1,) * 3, dtype=F64, device="cuda", generator=g))
        s["values"] = _fe27(m, kappa)[2]
    if kind == "adjoint":
        # the setup's operator, scaled a few per cent per unknown on both
        # sides: the coefficients of one optimisation step
        scale = 1.0 + 0.05 * uniform(n)
        v, rp, ci = (torch.as_tensor(np.asarray(plan.A[k]), device="cuda") for k in (3, 1, 2))
        rows = torch.repeat_interleave(torch.arange(n, device="cuda"), rp.long().diff())
        s["values"] = (v * scale[rows] * scale[ci.long()]).requires_grad_(True)
        s["b"].requires_grad_(True)
        s["w"] = uniform(n)
    torch.cuda.synchronize()
    return s


def run(s):
    case, plan = s["case"], s["plan"]
    h, cfg, kind, x, b = plan.h, plan.config, case["kind"], s["x"], s["b"]
    with torch.cuda.stream(plan.stream):
        if kind == "cycle":
            x.copy_(s["x0"])
            return draugr.amg_cycle(x, b, h, cfg)
        if kind == "resetup":
            draugr.amg_resetup(h, s["values"], cfg)
            x.copy_(s["x0"])
            return draugr.amg_cycle(x, b, h, cfg)
        if kind == "adjoint":
            y = draugr.amg_solve_diff(s["values"], b, h, cfg, tol=1e-10, precision=case["precision"],
                                      symmetric=case["problem"] == "het3d")
            gv, gb = torch.autograd.grad(y, (s["values"], b), s["w"])
            return {"x": y.detach(), "grad_values": gv, "grad_b": gb}
        x.zero_()
        if kind == "solve":
            return draugr.amg_solve(x, b, h, cfg)[0]
        if kind == "pcg":
            return draugr.pcg(x, b, h, cfg, precision=case["precision"])[0]
        if kind == "fgmres":
            return draugr.fgmres(x, b, h, cfg, precision=case["precision"])[0]
        if kind == "block":
            return draugr.pcg_multi(x, b, h, cfg, precision=case["precision"])[0]
        return draugr.pcg_batched(x, b, h, cfg, precision=case["precision"])[0]


# ------------------------------------------------------------ work

def _iterations(case):
    """Iterations the method takes on this case (the same for every correct
    implementation, give or take one): [forward, backward]."""
    s = prepare(case, 1)
    plan, kind, prec = s["plan"], case["kind"], case["precision"]
    h, cfg, x, b = plan.h, plan.config, s["x"], s["b"]
    with torch.no_grad(), torch.cuda.stream(plan.stream):
        x.zero_()
        if kind == "solve":
            return [draugr.amg_solve(x, b, h, cfg)[1]]
        if kind == "pcg":
            return [draugr.pcg(x, b, h, cfg, precision=prec)[1]]
        if kind == "fgmres":
            return [draugr.fgmres(x, b, h, cfg, precision=prec)[1]]
        if kind == "block":
            return [max(draugr.pcg_multi(x, b, h, cfg, precision=prec)[1])]
        if kind == "batch":
            return [int(np.mean(draugr.pcg_batched(x, b, h, cfg, precision=prec)[1]))]
        f = draugr.pcg if case["problem"] == "het3d" else draugr.bicgstab
        kw = {"tol": 1e-10, "precision": prec}
        draugr.amg_resetup(h, s["values"].detach(), cfg)
        first = f(x, b.detach(), h, cfg, **kw)[1]
        x.zero_()
        if f is draugr.bicgstab:
            kw["transpose"] = True
        return [first, f(x, s["w"], h, cfg, **kw)[1]]


def _cycle_work(case, h, zero_start, k=1):
    """Bytes and operations of one cycle: every level matrix once per
    smoothing step or residual that needs it (a first Jacobi step from zero
    needs none), P and its transpose once each, the level's vectors."""
    v = 4 if case["precision"] == "mixed" else 8
    sm = case["smoother"]
    step = CHEB_DEGREE if sm == "chebyshev" else 1
    nbytes = flops = 0
    for l in range(h.nlevels):
        n, nnz, nc, pnnz = (int(t) for t in h.level_info(l)[:4])
        free = 1 if sm in JACOBI_TYPE and (zero_start or l > 0) else 0
        passes = 2 * step + 1 - free
        visits = 2 ** l if case["cycle"] == "W" else 1
        nbytes += visits * (passes * ((4 + v) * nnz + 4 * n + 3 * v * n * k)
                            + 2 * ((4 + v) * pnnz + v * (n + nc) * k))
        flops += visits * k * (2 * passes * nnz + 4 * pnnz + 6 * passes * n)
    return nbytes, flops


def work(case):
    h, kind, k = _plan(case).h, case["kind"], case["k"]
    n, nnz = int(h.level_info(0)[0]), int(h.level_info(0)[1])
    if kind in ("cycle", "resetup"):
        nbytes, flops = _cycle_work(case, h, False)
        if kind == "resetup":
            # A, P and R read once, every coarse matrix written once
            for l in range(h.nlevels):
                _, lnnz, _, pnnz = (int(t) for t in h.level_info(l)[:4])
                after = int(h.level_info(l + 1 if l + 1 < h.nlevels else -1)[1])
                nbytes += 12 * lnnz + 24 * pnnz + 12 * after
                ap = int(h.level_info(l)[6])
                flops += 4 * max(ap, 0) + 4 * after
        return {"bytes": nbytes, "flops": flops}
    rhs = k if kind == "block" else 1
    cb, cf = _cycle_work(case, h, kind != "solve", rhs)
    # the outer product with A and the iteration's vectors
    per_b = cb + 12 * nnz + 4 * n + 8 * 10 * n * rhs
    per_f = cf + rhs * (2 * nnz + 12 * n)
    its = _iterations(case)
    total = sum(its)
    if kind == "adjoint" and case["problem"] != "het3d":
        total *= 2  # two cycles and two products per BiCGStab iteration
    nbytes, flops = total * per_b, total * per_f
    if kind == "adjoint":
        nbytes += 8 * 3 * nnz
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    """Cycles and resetups: about four times the error of sums in another
    order (1e-16 to 1e-14 for cycles, 4e-14 for a resetup against exact()),
    with room for hierarchies of other sizes.  Solves stop at a relative
    residual, so two correct implementations may stop an iteration apart:
    four times the error of the stopped iterate against exact()."""
    kind = case["kind"]
    if kind in ("cycle", "solve"):
        return {"rel": 1e-13}
    if kind == "resetup":
        return {"rel": 1e-12}
    return {"rel": {"fgmres": 2e-6, "batch": 2e-7}.get(kind, 1e-8)}


# ------------------------------------------------------------ 64-bit results

def _csr(n, m, rp, ci, v):
    return torch.sparse_csr_tensor(torch.as_tensor(np.asarray(rp, np.int64), device="cuda"),
                                   torch.as_tensor(np.asarray(ci, np.int64), device="cuda"),
                                   torch.as_tensor(np.asarray(v, np.float64), device="cuda"), size=(n, m))


def _transposed(M):
    return M.to_sparse_coo().t().coalesce().to_sparse_csr()


def _levels(case, h, values=None):
    """The hierarchy's operators as torch matrices; with `values`, rebuilt
    from new values of the finest matrix (P kept)."""
    out, A = [], None
    for l in range(h.nlevels):
        n, _, nc = (int(t) for t in h.level_info(l)[:3])
        if values is None or l == 0:
            v = h.export(l, "A_nzval") if values is None else values.detach().cpu().numpy()
            A = _csr(n, n, h.export(l, "A_rowptr"), h.export(l, "A_colval"), v)
        P = _csr(n, nc, h.export(l, "P_rowptr"), h.export(l, "P_colval"), h.export(l, "P_nzval"))
        lev = {"A": A, "P": P, "R": _transposed(P), "omega": float(h.export(l, "omega")[0])}
        if values is None:
            lev["d"] = torch.as_tensor(h.export(l, "invdiag"), device="cuda")
        else:
            lev["d"] = 1.0 / _rowsum_abs(A)
        if case["smoother"].endswith("colored_gs"):
            order, off = h.export(l, "color_order"), h.export(l, "color_offsets")
            lev["colors"] = [_rows_of(A, order[off[c]:off[c + 1]]) for c in range(len(off) - 1)]
        if case["smoother"] == "chebyshev":
            lev["cheb"] = h.export(l, "cheb_coef")
        out.append(lev)
        if values is not None:
            A = torch.sparse.mm(lev["R"], torch.sparse.mm(A, P))
    if values is None:
        nc = int(h.level_info(-1)[0])
        dense = torch.as_tensor(h.export(-1, "C_dense"), device="cuda").reshape(nc, nc).t()
    else:
        dense = A.to_dense()
    return out, torch.linalg.inv(dense)


def _rowsum_abs(A):
    rows = torch.repeat_interleave(torch.arange(A.shape[0], device="cuda"), A.crow_indices().diff())
    return torch.zeros(A.shape[0], dtype=F64, device="cuda").index_add_(0, rows, A.values().abs())


def _rows_of(A, rows):
    """(row indices, the matrix of those rows)."""
    rows = torch.as_tensor(np.asarray(rows, np.int64), device="cuda")
    rp = A.crow_indices()
    lens = rp[rows + 1] - rp[rows]
    nrp = torch.zeros(len(rows) + 1, dtype=torch.int64, device="cuda")
    nrp[1:] = torch.cumsum(lens, 0)
    k = torch.arange(int(nrp[-1]), device="cuda")
    k = k - torch.repeat_interleave(nrp[:-1], lens) + torch.repeat_interleave(rp[rows], lens)
    return rows, torch.sparse_csr_tensor(nrp, A.col_indices()[k], A.values()[k], size=(len(rows), A.shape[1]))


def _smooth(case, lev, x, b):
    d = lev["d"][:, None]
    if "colors" in lev:
        x = x.clone()
        for rows, sub in lev["colors"]:
            x[rows] += d[rows] * (b[rows] - sub @ x)
        return x
    if "cheb" in lev:
        c = lev["cheb"]
        p = None
        for j in range(len(c) // 2):
            r = b - lev["A"] @ x
            p = d * r * c[0] if j == 0 else c[2 * j] * d * r + c[2 * j + 1] * p
            x = x + p
        return x
    w = 1.0 if case["smoother"] == "spai0" else lev["omega"]
    return x + w * d * (b - lev["A"] @ x)


def _cycle(case, levels, cinv, x, b, l=0):
    if l == len(levels):
        return cinv @ b
    lev = levels[l]
    x = _smooth(case, lev, x, b)
    bc = lev["R"] @ (b - lev["A"] @ x)
    xc = _cycle(case, levels, cinv, torch.zeros_like(bc), bc, l + 1)
    if case["cycle"] == "W" and l + 1 < len(levels):
        xc = _cycle(case, levels, cinv, xc, bc, l + 1)
    x = x + lev["P"] @ xc
    return _smooth(case, lev, x, b)


def _solution(A, precond, b, rounds=3, maxiter=250):
    """A^-1 b for the columns of b: BiCGStab inside refinement, to rounding."""
    x = torch.zeros_like(b)
    bn = b.norm(dim=0).clamp_min(1e-300)
    safe = lambda t: torch.where(t == 0, torch.ones_like(t), t)
    for _ in range(rounds):
        r0 = b - A @ x
        if bool((r0.norm(dim=0) < 1e-15 * bn).all()):
            break
        dx, r = torch.zeros_like(b), r0.clone()
        p = v = torch.zeros_like(b)
        rho = alpha = omega = torch.ones(b.shape[1], dtype=F64, device="cuda")
        target = 1e-9 * r0.norm(dim=0)
        for _ in range(maxiter):
            rho1 = (r0 * r).sum(0)
            p = r + (rho1 / safe(rho)) * (alpha / safe(omega)) * (p - omega * v)
            ph = precond(p)
            v = A @ ph
            alpha = rho1 / safe((r0 * v).sum(0))
            s = r - alpha * v
            sh = precond(s)
            t = A @ sh
            omega = (t * s).sum(0) / safe((t * t).sum(0))
            dx = dx + alpha * ph + omega * sh
            r = s - omega * t
            rho = rho1
            if bool((r.norm(dim=0) < target).all()):
                break
        x = x + dx
    return x


def _diag_precond(A):
    rows = torch.repeat_interleave(torch.arange(A.shape[0], device="cuda"), A.crow_indices().diff())
    on = A.col_indices() == rows
    d = torch.ones(A.shape[0], dtype=F64, device="cuda")
    d[rows[on]] = A.values()[on]
    return lambda r: r / d[:, None]


def exact(case, seed):
    s = prepare(case, seed)
    plan, kind = s["plan"], case["kind"]
    h, b = plan.h, s["b"].detach()
    col = b if b.dim() == 2 else b[:, None]
    if kind == "batch":
        outs = []
        for A, off in zip(plan.mats, plan.h.offsets):
            M = _csr(*A.shape, A.indptr, A.indices, A.data)
            outs.append(_solution(M, _diag_precond(M), col[int(off):int(off) + A.shape[0]], maxiter=600))
        return torch.cat(outs)[:, 0]
    levels, cinv = _levels(case, h, s["values"] if kind == "resetup" else None)
    if kind in ("cycle", "resetup"):
        return _cycle(case, levels, cinv, s["x0"][:, None], col)[:, 0]
    if kind == "solve":
        x, bn = torch.zeros_like(col), col.norm()
        for _ in range(100):
            x = _cycle(case, levels, cinv, x, col)
            if float((col - levels[0]["A"] @ x).norm() / bn) < 1e-10:
                break
        return x[:, 0]
    A = levels[0]["A"]
    if kind == "adjoint":
        A = _csr(plan.n, plan.n, plan.A[1], plan.A[2], s["values"].detach().cpu().numpy())
    x = _solution(A, lambda r: _cycle(case, levels, cinv, torch.zeros_like(r), r), col)
    if kind != "adjoint":
        return x if b.dim() == 2 else x[:, 0]
    turned = [dict(lev, A=_transposed(lev["A"])) for lev in levels]
    At = _transposed(A)
    lam = _solution(At, lambda r: _cycle(case, turned, cinv.t(), torch.zeros_like(r), r), s["w"][:, None])[:, 0]
    x = x[:, 0]
    rows = torch.repeat_interleave(torch.arange(plan.n, device="cuda"), A.crow_indices().diff())
    return {"x": x, "grad_values": -lam[rows] * x[A.col_indices()], "grad_b": lam}
