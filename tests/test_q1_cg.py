"""The one-kernel CG of the Q1 operator against the oracle's CG on the oracle's
operator, over grids of one CTA, ragged ranges, and several vertices a thread."""
import ctypes as C

import numpy as np
import pytest


def _rhs(cells, seed):
    f = np.random.default_rng(seed).uniform(-1.0, 1.0, (cells[1] + 1, cells[0] + 1))
    f[[0, -1]] = 0.0
    f[:, [0, -1]] = 0.0
    return f.ravel()


def _exact(cells, f):
    """-lap u + u with Q1 elements, diagonalised by the sine modes."""
    def parts(n):
        i = np.arange(1, n)
        c = np.cos(np.pi * i / n)
        return np.sin(np.pi / n * np.outer(i, i)) * np.sqrt(2.0 / n), 2 * n * (1 - c), (2 + c) / (3.0 * n)
    (sy, ky, my), (sx, kx, mx) = parts(cells[1]), parts(cells[0])
    g = f.reshape(cells[1] + 1, cells[0] + 1)
    u = np.zeros_like(g)
    lam = np.outer(ky, mx) + np.outer(my, kx) + np.outer(my, mx)
    u[1:-1, 1:-1] = sy @ ((sy @ g[1:-1, 1:-1] @ sx) / lam) @ sx
    return u.ravel()


@pytest.mark.gpu
@pytest.mark.parametrize("diagonal", [True, False])
@pytest.mark.parametrize("cells", [(1, 1), (2, 2), (7, 3), (3, 90), (64, 64), (61, 77), (200, 131)])
def test_solution_and_iterations(gb, orc, cells, diagonal):
    """Relative residual 1e-12 in the energy of the stop: the solution within
    1e-9 (the condition number of these systems is below 1e5, times 1e-12 and
    the norms' ratio); the oracle's iteration count within 2 %, the rounding of
    the scalar products moving where the residual drops below."""
    op = gb.Q1Operator(cells, diffusion=1.0, mass=1.0)
    f = _rhs(cells, 5)
    pc = gb.Preconditioner.diagonal(op) if diagonal else None
    u = gb.DeviceArray(op.size)
    u.clear()
    inv = gb.KrylovInverseOperator("cg", tolerance=1e-12)
    inv.bind(op, pc)
    inv(gb.DeviceArray.from_numpy(f), u)
    info, ref = inv.info(), _exact(cells, f)
    assert info["converged"]
    assert np.max(np.abs(u.numpy() - ref)) <= 1e-9 * max(np.max(np.abs(ref)), 1e-300)
    if cells[0] * cells[1] < 6000:
        dg = orc.q1_apply(cells, None, 1.0, 1.0, diag_only=True)
        it, _, _ = orc.cg(lambda x: orc.q1_apply(cells, x, 1.0, 1.0), f, prec=(lambda r: r / dg) if diagonal else None,
                          epsilon=1e-12, max_iter=10000)
        assert abs(info["iterations"] - it) <= max(2, it // 50)


@pytest.mark.gpu
def test_start_vector_precision_and_stops(gb):
    """From a start vector (Dirichlet values kept), in FP32, capped, and with a
    tolerance that cannot be reached over more than one launch."""
    cells = (40, 33)
    f, ref = _rhs(cells, 7), _exact(cells, _rhs(cells, 7))
    op = gb.Q1Operator(cells, diffusion=1.0, mass=1.0)
    pc = gb.Preconditioner.diagonal(op)
    fd = gb.DeviceArray.from_numpy(f)
    inv = gb.KrylovInverseOperator("cg", tolerance=1e-12)
    inv.bind(op, pc)
    u = gb.DeviceArray.from_numpy(ref)
    inv(fd, u)
    assert inv.info()["converged"] and inv.info()["iterations"] <= 2
    op32 = gb.Q1Operator(cells, diffusion=1.0, mass=1.0, precision=gb.F32)
    pc32 = gb.Preconditioner.diagonal(op32)
    u32 = gb.DeviceArray(op32.size, gb.F32)
    u32.clear()
    inv = gb.KrylovInverseOperator("cg", tolerance=1e-5)
    inv.bind(op32, pc32)
    inv(gb.DeviceArray.from_numpy(f.astype(np.float32)), u32)
    assert inv.info()["converged"]
    assert np.max(np.abs(u32.numpy() - ref)) <= 1e-3 * np.max(np.abs(ref))
    u.clear()
    inv = gb.KrylovInverseOperator("cg", tolerance=1e-12, max_iterations=5)
    inv.bind(op, pc)
    inv(fd, u)
    assert inv.info()["iterations"] == -5 and not inv.info()["converged"]
    u.clear()
    inv = gb.KrylovInverseOperator("cg", tolerance=0.0, max_iterations=20000, error_measure=gb.ABSOLUTE)
    inv.bind(op, pc)
    inv(fd, u)
    info = inv.info()
    assert info["iterations"] == -20000 or info["residual"] == 0.0 or info["status"] != 0
    assert np.max(np.abs(u.numpy() - ref)) <= 1e-9 * np.max(np.abs(ref))


def _selftest(gb, op, pc, f, u, late_cta, no_cluster, no_grid=0, **kw):
    prm, info = gb.solver_params("cg", 1e-12, **kw), gb.SolverInfo()
    rc = gb.lib().gbfem_selftest_q1_cg(op.handle, pc.handle, C.byref(prm), f.ptr, u.ptr, C.byref(info),
                                       C.c_int(late_cta), C.c_int(no_cluster), C.c_int(no_grid))
    return rc, info


@pytest.mark.gpu
@pytest.mark.parametrize("late_cta", [0, 3, 5])
@pytest.mark.parametrize("iterations", [0, 50])
def test_a_block_that_gives_up_is_an_error(gb, late_cta, iterations):
    """Whichever block it is and whenever: without iterations the other blocks get
    all parts of the only sum and end as if all were well.  The next solve is
    unaffected."""
    cells = (40, 33)  # 1394 vertices, 6 blocks
    f, ref = _rhs(cells, 7), _exact(cells, _rhs(cells, 7))
    op = gb.Q1Operator(cells, diffusion=1.0, mass=1.0)
    pc = gb.Preconditioner.diagonal(op)
    fd, u = gb.DeviceArray.from_numpy(f), gb.DeviceArray(op.size)
    u.clear()
    kw = dict(error_measure=gb.ABSOLUTE, max_iterations=iterations)
    rc, _ = _selftest(gb, op, pc, fd, u, late_cta, 1, **kw)
    assert rc != 0
    u.clear()
    assert _selftest(gb, op, pc, fd, u, -1, 1, **kw)[0] == 0
    u.clear()
    rc, info = _selftest(gb, op, pc, fd, u, -1, 1)
    assert rc == 0 and info.converged
    assert np.max(np.abs(u.numpy() - ref)) <= 1e-9 * np.max(np.abs(ref))


@pytest.mark.gpu
@pytest.mark.parametrize("cells", [(1, 1), (7, 3), (64, 64)])
@pytest.mark.parametrize("no_cluster,no_grid", [(0, 0), (1, 0), (1, 1)])
def test_where_the_device_cannot_place_it(gb, cells, no_cluster, no_grid):
    """Without room for a cluster the other form, without room for that the general
    loop: the same solution, and as many iterations within 2 %."""
    f, ref = _rhs(cells, 3), _exact(cells, _rhs(cells, 3))
    op = gb.Q1Operator(cells, diffusion=1.0, mass=1.0)
    pc = gb.Preconditioner.diagonal(op)
    fd, u, its = gb.DeviceArray.from_numpy(f), gb.DeviceArray(op.size), []
    for forms in ((0, 0), (no_cluster, no_grid)):
        u.clear()
        rc, info = _selftest(gb, op, pc, fd, u, -1, *forms)
        assert rc == 0 and info.converged
        assert np.max(np.abs(u.numpy() - ref)) <= 1e-9 * max(np.max(np.abs(ref)), 1e-300)
        its.append(info.iterations)
    assert abs(its[0] - its[1]) <= max(2, its[0] // 50)
