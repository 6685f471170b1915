"""Performance cases: the calls a program that uses this library spends its time in.

listed() is a fixed selection, draw(rng) gives more of the same ranges.  Every
case goes through the public Python binding (dune-fem_gb300/gbfem.py):

  apply        w = A u, the SIPG / upwind / mass operator on a hexahedral grid:
               constant or cellwise kappa (closed form) or kappa a DG field
               (Gauss-point quadrature), FP64 and FP32
  host_apply   the same from page-locked host buffers, copies included
  rk3          one explicit SSP-RK3 step of the advection-diffusion operator
  linearise    the body of a Newton step: residual, Jacobian at u, Jacobian apply
  scaled_bj    the mixed solve's preconditioner apply (FP32)
  block_jacobi the FP64 CG's preconditioner apply
  q1cg         the whole 2-D Q1 Poisson-type solve, CG with diagonal preconditioner
  mixed        the whole variable-kappa solve, FP32 CG inside FP64 FGMRES
  cnn          the learned preconditioner's network, r -> z

exact() evaluates the same forms in plain FP64 torch: at the Gauss points for
the operators (exact for the polynomial integrands), by sine transforms for
the Q1 solve, by dense cell blocks for the preconditioners.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "dune-fem_gb300"))
import gbfem  # noqa: E402

DEV = "cuda"
VELOCITY = (1.0, 0.5, 0.25)


def listed():
    return [
        # the headline workload: every operator apply of an FP64 Krylov solve with constant coefficients
        {"name": "apply_q3_f64_64", "kind": "apply", "nx": 64, "ny": 64, "nz": 64, "order": 3, "f32": False,
         "coef": "const", "advect": False},
        # a unit-test / coarse-grid sized apply: the time of one call
        {"name": "apply_q2_f64_small", "kind": "apply", "nx": 6, "ny": 5, "nz": 7, "order": 2, "f32": False,
         "coef": "const", "advect": True},
        # the FP64 operator of a variable-coefficient solve (outer residuals, FP64 CG), ragged grid
        {"name": "apply_kappa_q3_f64", "kind": "apply", "nx": 45, "ny": 38, "nz": 33, "order": 3, "f32": False,
         "coef": "field", "advect": False},
        # the inner operator of the mixed solve: FP32, kappa per cell
        {"name": "apply_kcell_q3_f32_64", "kind": "apply", "nx": 64, "ny": 64, "nz": 64, "order": 3, "f32": True,
         "coef": "cell", "advect": False},
        # a call from a host program that keeps its dof vectors in its own memory
        {"name": "host_apply_q3_f64_64", "kind": "host_apply", "nx": 64, "ny": 64, "nz": 64, "order": 3},
        # explicit time stepping of periodic advection-diffusion
        {"name": "rk3_q2_f64_80", "kind": "rk3", "nx": 80, "ny": 80, "nz": 80, "order": 2, "f32": False},
        # one Newton step's operator work on the Bratu problem
        {"name": "linearise_q2_f64", "kind": "linearise", "nx": 32, "ny": 32, "nz": 32, "order": 2},
        # the preconditioner of the mixed solve at its highest order
        {"name": "scaled_bj_q4_f32_48", "kind": "scaled_bj", "nx": 48, "ny": 48, "nz": 48, "order": 4},
        # the preconditioner of the FP64 solve (dense cell blocks)
        {"name": "block_jacobi_q2_f64", "kind": "block_jacobi", "nx": 40, "ny": 36, "nz": 33, "order": 2},
        # the reference's introductory 2-D problem, whole solve
        {"name": "q1cg_64", "kind": "q1cg", "nx": 64, "ny": 64, "chunk": 32},
        # the variable-coefficient solve to 1e-10, whole
        {"name": "mixed_q3_32", "kind": "mixed", "nx": 32, "ny": 32, "nz": 32, "order": 3},
        # the learned preconditioner's network
        {"name": "cnn_q3_32", "kind": "cnn", "n": 32, "order": 3},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


# cells of the largest grid of each order: about 17 million dofs, as the headline grid
_MOST_CELLS = {1: 2000000, 2: 600000, 3: 262144, 4: 130000}


def _grid(rng, least, most):
    """nx, ny, nz: about a log-uniform number of cells, the sides unequal and often odd."""
    cells = _log_int(rng, least, most)
    side = cells ** (1.0 / 3.0)
    nx = max(2, int(side * rng.uniform(0.7, 1.2)))
    ny = max(2, int(side * rng.uniform(0.7, 1.2)))
    nz = max(2, min(int(cells / (nx * ny)), int(2 * side)))
    return {"nx": nx, "ny": ny, "nz": nz}


def draw(rng):
    kind = rng.choice(["apply"] * 5 + ["host_apply", "rk3", "linearise", "scaled_bj", "block_jacobi", "q1cg", "mixed",
                                       "cnn"])
    if kind == "apply":
        order = rng.choice([1, 2, 3, 3, 4])
        coef = rng.choice(["const", "const", "field", "cell"])
        return {"kind": kind, **_grid(rng, 100, _MOST_CELLS[order] / (1 if coef != "field" else 4)), "order": order,
                "f32": rng.random() < 0.4, "coef": coef, "advect": coef == "const" and rng.random() < 0.4}
    if kind == "host_apply":
        order = rng.choice([2, 3])
        return {"kind": kind, **_grid(rng, 1000, _MOST_CELLS[order]), "order": order}
    if kind == "rk3":
        order = rng.choice([1, 2, 3])
        return {"kind": kind, **_grid(rng, 200, _MOST_CELLS[order] / 2), "order": order, "f32": rng.random() < 0.5}
    if kind == "linearise":
        order = rng.choice([1, 2, 3])
        return {"kind": kind, **_grid(rng, 100, _MOST_CELLS[order] / 10), "order": order}
    if kind == "scaled_bj":
        order = rng.choice([2, 3, 4])
        return {"kind": kind, **_grid(rng, 500, _MOST_CELLS[order]), "order": order}
    if kind == "block_jacobi":
        order = rng.choice([1, 2, 3])
        return {"kind": kind, **_grid(rng, 200, _MOST_CELLS[order] / 10), "order": order}
    if kind == "q1cg":
        return {"kind": kind, "nx": _log_int(rng, 17, 150), "ny": _log_int(rng, 17, 150), "chunk": rng.choice([0, 32])}
    if kind == "mixed":
        order = rng.choice([2, 3])
        return {"kind": kind, **_grid(rng, 300, 24000), "order": order}
    return {"kind": kind, "n": rng.choice([8, 16, 24, 40]), "order": rng.choice([2, 3])}


# ---- inputs ---------------------------------------------------------------------------------------------------


def _cells(c):
    return (c["nx"], c["ny"], c["nz"])


def _uniform(n, seed, salt, f32=False):
    g = torch.Generator(device=DEV)
    g.manual_seed(1000003 * salt + seed)
    return torch.rand(n, generator=g, device=DEV, dtype=torch.float64).mul_(2.0).sub_(1.0).to(
        torch.float32 if f32 else torch.float64)


def _device(t):
    """A dof vector of the library with the values of t."""
    a = gbfem.DeviceArray(t.numel(), gbfem.F32 if t.dtype == torch.float32 else gbfem.F64)
    a.as_tensor().copy_(t.reshape(-1))
    return a


def _log_field(points, seed, modes=64, corr=0.1):
    """A Gaussian random field (std 1) from random Fourier modes at the tensor grid of the 1-D point lists
    (x, y, z): values [z][y][x]."""
    r = np.random.default_rng(seed)
    k = torch.from_numpy(r.normal(0.0, 1.0 / corr, (modes, 3))).to(DEV)
    phase = torch.from_numpy(r.uniform(0.0, 2.0 * math.pi, modes)).to(DEV)
    e = [torch.polar(torch.ones_like(p[:, None] * k[:, d]), p[:, None] * k[:, d]) for d, p in enumerate(points)]
    yz = e[2][:, None, :] * e[1][None, :, :]
    x = e[0] * torch.polar(torch.ones_like(phase), phase)
    return (yz.reshape(-1, modes) @ x.T).real.mul(math.sqrt(2.0 / modes)).reshape(
        e[2].shape[0], e[1].shape[0], e[0].shape[0])


def _points(cells, pts):
    return [((torch.arange(n, device=DEV, dtype=torch.float64)[:, None] + pts) / n).reshape(-1) for n in cells]


def _at_cells(v, cells, q):
    """[z q][y q][x q] point values as [z][y][x][a][b][c], (a, b, c) along x, y, z."""
    nx, ny, nz = cells
    return v.reshape(nz, q, ny, q, nx, q).permute(0, 2, 4, 5, 3, 1)


def _kappa_field(cells, order, seed):
    """exp of a Gaussian field, projected onto the DG space: coefficients [z][y][x][i][j][k]."""
    t = _Tables(order + 1, order + 2)
    v = _at_cells(torch.exp(_log_field(_points(cells, t.x), seed)), cells, t.q)
    for d in range(3):
        v = _along(v, t.B.T * t.w, d)
    return v.contiguous()


def _kappa_cells(cells, seed):
    mid = torch.full((1,), 0.5, device=DEV, dtype=torch.float64)
    return torch.exp(_log_field(_points(cells, mid), seed)).to(torch.float32)


def _bump(cells, order, seed, f32):
    """A Gaussian bump of width 0.1 near the centre, projected onto the DG space."""
    t = _Tables(order + 1, order + 2)
    centre = 0.5 + 0.1 * (np.random.default_rng(seed).random(3) - 0.5)
    f = []
    for d, p in enumerate(_points(cells, t.x)):
        e = torch.exp(-((p - float(centre[d])) / 0.1) ** 2).reshape(cells[d], t.q)
        f.append(e @ (t.B * t.w[:, None]))
    return torch.einsum("xi,yj,zk->zyxijk", f[0], f[1], f[2]).to(torch.float32 if f32 else torch.float64)


_RK = dict(diffusion=1e-3, velocity=VELOCITY, periodic=(1, 1, 1), weak_dirichlet=False)
_BRATU = (0.0, 0.0, -5.0)


def _time_step(cells, order):
    """CFL 0.2 of the advective step, below the stability bound of the interior-penalty diffusion."""
    adv = 0.2 / (max(cells) * math.sqrt(sum(v * v for v in VELOCITY)) * (2 * order + 1))
    dif = 0.5 / (4.0 * 1e-3 * 10.0 * (order + 1) ** 4 * sum(n * n for n in cells))
    return min(adv, dif)


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind}
    if kind == "q1cg":
        s["f"] = _device(_q1_rhs(case, seed))
        s["op"] = gbfem.Q1Operator((case["nx"], case["ny"]), diffusion=1.0, mass=1.0)
        s["u"] = gbfem.DeviceArray(s["op"].size)
        s["inv"] = gbfem.KrylovInverseOperator("cg", tolerance=1e-10, graph_chunk=case["chunk"])
        s["inv"].bind(s["op"], gbfem.Preconditioner.diagonal(s["op"]))
        return s
    if kind == "cnn":
        n, order = case["n"], case["order"]
        cells, nloc = (n, n, n), (order + 1) ** 3
        s["net"] = gbfem.CNN(order, n, seed=1)
        s["net"].set_kappa(_device(_kappa_field(cells, order, seed)))
        s["r"] = _device(_uniform(n ** 3 * nloc, seed, 1))
        s["z"] = gbfem.DeviceArray(n ** 3 * nloc)
        return s
    cells, order = _cells(case), case["order"]
    n = cells[0] * cells[1] * cells[2] * (order + 1) ** 3
    if kind == "apply":
        f32 = case["f32"]
        prec = gbfem.F32 if f32 else gbfem.F64
        kw = dict(precision=prec)
        if case["coef"] == "field":
            k = _kappa_field(cells, order, seed)
            kw["kappa"] = _device(k.to(torch.float32) if f32 else k)
        elif case["coef"] == "cell":
            k = _kappa_cells(cells, seed)
            kw["kappa_cell"] = _device(k if f32 else k.double())
        elif case["advect"]:
            kw.update(diffusion=1e-2, velocity=VELOCITY, mass=1.0)
        s["op"] = gbfem.DGOperator(cells, order, **kw)
        s["u"] = _device(_uniform(n, seed, 1, f32))
        s["w"] = gbfem.DeviceArray(n, prec)
    elif kind == "host_apply":
        s["op"] = gbfem.DGOperator(cells, order)
        s["pin"] = [_uniform(n, seed, 1).cpu().pin_memory(), torch.zeros(n, dtype=torch.float64).pin_memory()]
        s["u"], s["w"] = (t.numpy() for t in s["pin"])
    elif kind == "rk3":
        u = _bump(cells, order, seed, case["f32"])
        s["op"] = gbfem.DGOperator(cells, order, precision=gbfem.F32 if case["f32"] else gbfem.F64, **_RK)
        s["u"], s["rk"], s["dt"] = _device(u), gbfem.RK3(s["op"]), _time_step(cells, order)
    elif kind == "linearise":
        s["op"] = gbfem.NonlinearDGOperator(cells, order, reaction=_BRATU)
        s["u"], s["d"] = _device(0.3 * _uniform(n, seed, 1)), _device(_uniform(n, seed, 2))
        s["r"], s["w"] = gbfem.DeviceArray(n), gbfem.DeviceArray(n)
        s["jac"] = s["op"].jacobian(s["u"])
    elif kind == "scaled_bj":
        s["op"] = gbfem.DGOperator(cells, order, precision=gbfem.F32, kappa_cell=_device(_kappa_cells(cells, seed)))
        s["pc"] = gbfem.Preconditioner.scaled_block_jacobi(s["op"])
        s["r"], s["z"] = _device(_uniform(n, seed, 1, True)), gbfem.DeviceArray(n, gbfem.F32)
    elif kind == "block_jacobi":
        s["op"] = gbfem.DGOperator(cells, order, kappa=_device(_kappa_field(cells, order, seed)))
        s["pc"] = gbfem.Preconditioner.block_jacobi(s["op"])
        s["r"], s["z"] = _device(_uniform(n, seed, 1)), gbfem.DeviceArray(n)
    elif kind == "mixed":
        k = _kappa_field(cells, order, seed)
        f = torch.zeros_like(k)
        f[..., 0, 0, 0] = 1.0 / (cells[0] * cells[1] * cells[2])
        s["op"] = gbfem.DGOperator(cells, order, kappa=_device(k))
        mean = k[..., 0, 0, 0].to(torch.float32)
        s["op32"] = gbfem.DGOperator(cells, order, precision=gbfem.F32, kappa_cell=_device(mean))
        s["pc"] = gbfem.Preconditioner.scaled_block_jacobi(s["op32"])
        s["f"], s["u"] = _device(f), gbfem.DeviceArray(n)
    return s


def run(s):
    kind = s["kind"]
    if kind == "apply":
        s["op"](s["u"], s["w"])
        return s["w"].as_tensor()
    if kind == "host_apply":
        s["op"].apply_host(s["u"], s["w"])
        return s["w"]
    if kind == "rk3":
        s["rk"].step(s["u"], s["dt"])
        return s["u"].as_tensor()
    if kind == "linearise":
        s["op"](s["u"], s["r"])
        s["op"].jacobian(s["u"], s["jac"])
        s["jac"](s["d"], s["w"])
        return {"residual": s["r"].as_tensor(), "jacobian_apply": s["w"].as_tensor()}
    if kind in ("scaled_bj", "block_jacobi"):
        s["pc"](s["r"], s["z"])
        return s["z"].as_tensor()
    if kind == "cnn":
        s["net"].forward(s["r"], s["z"])
        return s["z"].as_tensor()
    s["u"].clear()
    if kind == "q1cg":
        s["inv"](s["f"], s["u"])
    else:
        gbfem.solve_mixed(s["op"], s["op32"], s["pc"], s["f"], s["u"], tolerance=1e-10, inner_tolerance=1e-2,
                          max_outer=300, outer="fgmres", outer_restart=30, graph_chunk=16)
    return s["u"].as_tensor()


def work(case):
    """Inputs read once, outputs written once; arithmetic of the cheapest known evaluation (per dof of a cell line:
    the closed form's line operators, or the sum-factorised contractions at q = p + 2 points)."""
    kind = case["kind"]
    if kind == "q1cg":
        nv = (case["nx"] + 1) * (case["ny"] + 1)
        its = 2.4 * math.sqrt(case["nx"] * case["ny"])  # about what CG takes on this problem
        return {"bytes": 16.0 * nv, "flops": its * 30.0 * nv}
    if kind == "cnn":
        n3, nloc = case["n"] ** 3, (case["order"] + 1) ** 3
        convs = 2 + 2.0 / 8 + 2.0 / 64 + 1.0 / 512
        return {"bytes": 16.0 * n3 * nloc, "flops": 2.0 * n3 * (27 * 32 * 32 * convs + 64.0 * nloc)}
    n1 = case["order"] + 1
    q = n1 + 1
    cells = case["nx"] * case["ny"] * case["nz"]
    n = float(cells * n1 ** 3)
    closed = n * (3.0 * (2 * n1 + 5) + 3.0)
    # volume: values 3 contractions, gradients 3, flux, the transposes; six faces of two traces each
    quad = cells * 2.0 * (2 * (q * n1 ** 3 + q * q * n1 * n1 + q ** 3 * n1) + 6 * q ** 4 + 8 * q ** 3
                          + 6 * (2 * n1 ** 3 + 6 * (q * n1 * n1 + q * q * n1) + 8 * q * q))
    if kind == "apply":
        es = 4.0 if case["f32"] else 8.0
        if case["coef"] == "field":
            return {"bytes": 3 * es * n, "flops": quad}
        return {"bytes": 2 * es * n, "flops": closed}
    if kind == "host_apply":
        return {"bytes": 16.0 * n, "flops": closed}
    if kind == "rk3":
        return {"bytes": 3 * 2 * (4.0 if case["f32"] else 8.0) * n, "flops": 3 * (closed + 6 * n)}
    if kind == "linearise":
        react = cells * 4.0 * (q * n1 ** 3 + q * q * n1 * n1 + q ** 3 * n1)
        return {"bytes": 4 * 8.0 * n, "flops": 2 * closed + 2.5 * react}
    if kind == "scaled_bj":
        return {"bytes": 8.0 * n, "flops": 2.0 * n * n1 ** 3}
    if kind == "block_jacobi":
        return {"bytes": 8.0 * n * (n1 ** 3 + 2), "flops": 2.0 * n * n1 ** 3}
    # mixed: kappa, f and u; about 120 inner iterations per cell of the longest side
    its = 120.0 * max(case["nx"], case["ny"], case["nz"])
    return {"bytes": 24.0 * n, "flops": its * (closed + 2.0 * n * n1 ** 3)}


# ---- the same in plain FP64 -----------------------------------------------------------------------------------


class _Tables:
    """Gauss points on [0, 1] and orthonormal Legendre values there and at 0 and 1."""

    def __init__(self, n, q):
        x, w = np.polynomial.legendre.leggauss(q)
        leg = np.polynomial.legendre
        scale = [math.sqrt(2 * i + 1) for i in range(n)]
        value = lambda t: np.stack([scale[i] * leg.legval(t, np.eye(n)[i]) for i in range(n)], -1)  # noqa: E731
        slope = lambda t: np.stack(  # noqa: E731
            [2 * scale[i] * leg.legval(t, leg.legder(np.eye(n)[i])) * np.ones_like(t) for i in range(n)], -1)
        ends = np.array([-1.0, 1.0])
        self.n, self.q = n, q
        self.x, self.w, self.B, self.G, self.tr, self.dtr = (
            torch.from_numpy(np.ascontiguousarray(v)).to(DEV) for v in
            (0.5 * (x + 1), 0.5 * w, value(x), slope(x), value(ends), slope(ends)))


def _along(v, m, d):
    """The matrix m applied along local axis d (of the last three) of v."""
    return torch.movedim(torch.tensordot(v, m, dims=([v.dim() - 3 + d], [1])), -1, v.dim() - 3 + d)


def _dg_apply(order, u, kappa=None, eps=1.0, mass=0.0, velocity=(0.0, 0.0, 0.0), periodic=False, weak=True, own=False,
              point=None):
    """The DG form applied to u [z][y][x][i][j][k] at q = p + 2 Gauss points.  kappa: None, a value per cell
    [z][y][x] or DG coefficients; own: neighbours' dofs taken as zero; point: a pointwise reaction of the values."""
    t = _Tables(order + 1, order + 2)
    n, q = t.n, t.q
    nc = (u.shape[2], u.shape[1], u.shape[0])
    vol = 1.0 / (nc[0] * nc[1] * nc[2])

    def kappa_at(mats):
        if kappa is None:
            return 1.0
        if kappa.dim() == 3:
            return kappa[..., None, None, None]
        v = kappa
        for d, m in enumerate(mats):
            v = _along(v, m, d)
        return v

    def interpolate(v, mats):
        for d, m in enumerate(mats):
            v = _along(v, m, d)
        return v

    W = vol * t.w[:, None, None] * t.w[None, :, None] * t.w[None, None, :]
    kq = kappa_at([t.B] * 3)
    val = interpolate(u, [t.B] * 3)
    src = mass * val
    if point is not None:
        src = src + point(val)
    w = interpolate(W * src, [t.B.T] * 3)
    for d in range(3):
        mats = [t.G if e == d else t.B for e in range(3)]
        flux = eps * kq * nc[d] * interpolate(u, mats) - velocity[d] * val
        w += interpolate(W * flux, [m.T for m in mats]) * nc[d]
        del flux
    del val, src, kq
    for d in range(3):
        h = 1.0 / nc[d]
        area = vol / h
        sigma = 10.0 * n * n / h
        ww = (t.w[:, None] * t.w[None, :] * area).reshape([1] * 3 + [1 if e == d else q for e in range(3)])
        ends = {}
        for s in (0, 1):
            vals, slopes = ([m[s:s + 1] if e == d else t.B for e in range(3)] for m in (t.tr, t.dtr))
            k = kappa_at(vals)
            ends[s] = (interpolate(u, vals), (1 if s else -1) / h * interpolate(u, slopes), k)
        for s in (0, 1):
            ax = 2 - d
            vm, dm, km = ends[s]
            vp, dp, kp = (x if not torch.is_tensor(x) else torch.roll(x, -1 if s else 1, ax) for x in ends[1 - s])
            edge = torch.zeros(nc[d], dtype=torch.bool, device=DEV)
            if not periodic:
                edge[nc[d] - 1 if s else 0] = True
            shape = [1] * 6
            shape[ax] = nc[d]
            edge = edge.reshape(shape)
            if own:
                vp, dp = torch.zeros_like(vp), torch.zeros_like(dp)
            bn = velocity[d] if s else -velocity[d]
            jump = vm - vp
            inner = eps * (sigma * 0.5 * (km + kp) * jump - 0.5 * (km * dm - kp * dp)) + bn * (vm if bn >= 0 else vp)
            outer = (eps * (sigma * km * vm - km * dm) if weak else 0.0 * vm) + max(bn, 0.0) * vm
            inner_g, outer_g = -0.5 * eps * km * jump, (-eps * km * vm if weak else 0.0 * vm)
            fv, fg = torch.where(edge, outer, inner) * ww, torch.where(edge, outer_g, inner_g) * ww
            w += interpolate(fv, [t.tr[s:s + 1].T if e == d else t.B.T for e in range(3)])
            w += interpolate(fg, [t.dtr[s:s + 1].T * ((1 if s else -1) / h) if e == d else t.B.T for e in range(3)])
    return w


def _shaped(v, cells, order):
    n = order + 1
    return v.double().reshape(cells[2], cells[1], cells[0], n, n, n)


def _q1_rhs(case, seed):
    """A random right-hand side that vanishes on the boundary."""
    f = _uniform((case["nx"] + 1) * (case["ny"] + 1), seed, 1).reshape(case["ny"] + 1, case["nx"] + 1)
    f[0], f[-1], f[:, 0], f[:, -1] = 0.0, 0.0, 0.0, 0.0
    return f


def _q1_solve(case, seed):
    f = _q1_rhs(case, seed)
    modes, stiff, mass = [], [], []
    for n in (case["ny"], case["nx"]):
        i = torch.arange(1, n, device=DEV, dtype=torch.float64)
        modes.append(torch.sin(math.pi / n * i[:, None] * i[None, :]) * math.sqrt(2.0 / n))
        c = torch.cos(math.pi / n * i)
        stiff.append(2.0 * n * (1.0 - c))
        mass.append((2.0 + c) / (3.0 * n))
    lam = stiff[0][:, None] * mass[1] + mass[0][:, None] * stiff[1] + mass[0][:, None] * mass[1]
    u = torch.zeros_like(f)
    u[1:-1, 1:-1] = modes[0] @ ((modes[0] @ f[1:-1, 1:-1] @ modes[1]) / lam) @ modes[1]
    return u


def _scaled_blocks(case, seed):
    """z = H^{-1} r / kappa with the kappa = 1 diagonal block of the cell's place in the grid."""
    cells, order = _cells(case), case["order"]
    n = order + 1
    t = _Tables(n, n + 1)
    vol = 1.0 / (cells[0] * cells[1] * cells[2])
    K = (t.G * t.w[:, None]).T @ t.G
    one = {}
    for d in range(3):
        h = 1.0 / cells[d]
        for low in (False, True):
            for high in (False, True):
                A = vol / h ** 2 * K
                for s, end in ((0, low), (1, high)):
                    v, g = t.tr[s], t.dtr[s] * ((1 if s else -1) / h)
                    c = 1.0 if end else 0.5
                    A = A + vol / h * (10.0 * n * n / h * torch.outer(v, v) - c * (torch.outer(v, g) + torch.outer(g, v)))
                one[d, low, high] = A
    eye = torch.eye(n, device=DEV, dtype=torch.float64)
    r = _shaped(_uniform(cells[0] * cells[1] * cells[2] * n ** 3, seed, 1, True), cells, order)
    z = torch.empty_like(r)
    spans = []
    for c in cells:
        spans.append([(slice(0, 1), c >= 1, c == 1)] + ([(slice(1, c - 1), False, False)] if c > 2 else [])
                     + ([(slice(c - 1, c), False, True)] if c > 1 else []))
    for sx, lx, hx in spans[0]:
        for sy, ly, hy in spans[1]:
            for sz, lz, hz in spans[2]:
                H = (torch.einsum("ai,bj,ck->abcijk", one[0, lx, hx], eye, eye)
                     + torch.einsum("ai,bj,ck->abcijk", eye, one[1, ly, hy], eye)
                     + torch.einsum("ai,bj,ck->abcijk", eye, eye, one[2, lz, hz])).reshape(n ** 3, n ** 3)
                b = r[sz, sy, sx].reshape(-1, n ** 3)
                z[sz, sy, sx] = torch.linalg.solve(H, b.T).T.reshape(r[sz, sy, sx].shape)
    return z / _kappa_cells(cells, seed).double()[..., None, None, None]


def exact(case, seed):
    kind = case["kind"]
    if kind in ("mixed", "cnn"):
        return None
    if kind == "q1cg":
        return _q1_solve(case, seed).reshape(-1)
    if kind == "scaled_bj":
        return _scaled_blocks(case, seed).reshape(-1)
    cells, order = _cells(case), case["order"]
    n = cells[0] * cells[1] * cells[2] * (order + 1) ** 3
    if kind == "apply":
        u = _shaped(_uniform(n, seed, 1, case["f32"]), cells, order)
        kw = {}
        if case["coef"] == "field":
            k = _kappa_field(cells, order, seed)
            kw["kappa"] = k.to(torch.float32).double() if case["f32"] else k
        elif case["coef"] == "cell":
            kw["kappa"] = _kappa_cells(cells, seed).double()
        elif case["advect"]:
            kw.update(eps=1e-2, velocity=VELOCITY, mass=1.0)
        return _dg_apply(order, u, **kw).reshape(-1)
    if kind == "host_apply":
        return _dg_apply(order, _shaped(_uniform(n, seed, 1), cells, order)).reshape(-1).cpu().numpy()
    if kind == "rk3":
        u = _bump(cells, order, seed, case["f32"]).double()
        f = -_time_step(cells, order) * cells[0] * cells[1] * cells[2]
        A = lambda v: f * _dg_apply(order, v, eps=1e-3, velocity=VELOCITY, periodic=True, weak=False)  # noqa: E731
        k0 = A(u)
        k1 = A(u + k0)
        k2 = A(u + 0.25 * (k0 + k1))
        return (u + (k0 + k1 + 4.0 * k2) / 6.0).reshape(-1)
    if kind == "linearise":
        u, d = (_shaped(s * _uniform(n, seed, k), cells, order) for s, k in ((0.3, 1), (1.0, 2)))
        t = _Tables(order + 1, order + 2)
        uq = u
        for e in range(3):
            uq = _along(uq, t.B, e)
        return {"residual": _dg_apply(order, u, point=lambda v: -5.0 * torch.exp(v)).reshape(-1),
                "jacobian_apply": _dg_apply(order, d, point=lambda v: -5.0 * torch.exp(uq) * v).reshape(-1)}
    # block_jacobi: the dense diagonal blocks, column by column
    n3 = (order + 1) ** 3
    k = _kappa_field(cells, order, seed)
    blocks = torch.empty(n // n3, n3, n3, device=DEV, dtype=torch.float64)
    for j in range(n3):
        e = torch.zeros(n // n3, n3, device=DEV, dtype=torch.float64)
        e[:, j] = 1.0
        blocks[:, :, j] = _dg_apply(order, _shaped(e, cells, order), kappa=k, own=True).reshape(-1, n3)
    return torch.linalg.solve(blocks, _uniform(n, seed, 1).reshape(-1, n3)).reshape(-1)
