"""The device-resident CG on more than one CTA: its fused FP32 products, the state
kept over a mixed solve's inner solves, and the general loop on the Q1 operator."""
import numpy as np
import pytest

from test_q1_cg import _rhs, _selftest


def _solve(gb, op, pc, f, tol, chunk):
    inv = gb.KrylovInverseOperator("cg", tolerance=tol, graph_chunk=chunk)
    inv.bind(op, pc)
    u = gb.DeviceArray(op.size, op.precision)
    u.clear()
    inv(f, u)
    return inv.info(), u.numpy()


@pytest.mark.gpu
@pytest.mark.parametrize("pc", [None, "diagonal", "block_jacobi"])
def test_fp64_iterates_equal_host_loop(gb, pc):
    """Sums of many CTAs, in the host loop's order: bit for bit."""
    op = gb.DGOperator((17, 15, 14), 2, mass=0.5)
    f = gb.DeviceArray.from_numpy(np.random.default_rng(1).uniform(-1, 1, op.size))
    p = getattr(gb.Preconditioner, pc)(op) if pc else None
    (ih, uh), (ig, ug) = (_solve(gb, op, p, f, 1e-10, chunk) for chunk in (0, 7))
    assert ih["converged"] and ig["iterations"] == ih["iterations"] and ig["residual"] == ih["residual"]
    assert np.array_equal(ug, uh)


@pytest.mark.gpu
@pytest.mark.parametrize("order,cells", [(1, (21, 9, 10)), (2, (11, 9, 9)), (3, (9, 9, 10)), (4, (7, 9, 9))])
@pytest.mark.parametrize("kcell", [True, False])
def test_fp32_iterates_close_to_host_loop(gb, order, cells, kcell):
    """The fused product sums <q, h> by bricks, compensated: alpha differs from the host
    loop's only where FP64's last bits decide its rounding to FP32, and the iterates
    then by FP32 rounding times the condition number, at most 1e4 here."""
    rng = np.random.default_rng(order)
    kw = dict(kappa_cell=gb.DeviceArray.from_numpy(rng.uniform(0.5, 2, np.prod(cells)).astype(np.float32))) if kcell else {}
    op = gb.DGOperator(cells, order, precision=gb.F32, **kw)
    f = gb.DeviceArray.from_numpy(rng.uniform(-1, 1, op.size).astype(np.float32))
    pc = gb.Preconditioner.block_jacobi(op)
    (ih, uh), (ig, ug) = (_solve(gb, op, pc, f, 1e-5, chunk) for chunk in (0, 16))
    assert ih["converged"] and ig["converged"] and abs(ig["iterations"] - ih["iterations"]) <= 2
    assert np.linalg.norm(ug - uh) <= 1e4 * 2.0 ** -24 * np.linalg.norm(uh)


@pytest.mark.gpu
@pytest.mark.parametrize("outer", ["fgmres", "refinement"])
@pytest.mark.parametrize("order,cells", [(1, (21, 9, 10)), (2, (11, 9, 9)), (3, (9, 9, 10)), (4, (7, 9, 9))])
def test_mixed_solve_equals_host_loop(gb, order, cells, outer):
    """Several inner solves with one state (vectors, graph): as with the host loop, the
    solutions within 1e-9 (true residuals of 1e-10 and a condition number whose square
    root is about 100), the inner iterations within 5 %."""
    nc, nloc = int(np.prod(cells)), (order + 1) ** 3
    rng = np.random.default_rng(order)
    k = np.zeros((nc, nloc))
    k[:, 0], k[:, 1] = rng.uniform(0.5, 2, nc), rng.uniform(-0.1, 0.1, nc)
    f = gb.DeviceArray.from_numpy(rng.uniform(-1, 1, nc * nloc))
    op = gb.DGOperator(cells, order, kappa=gb.DeviceArray.from_numpy(k.ravel()))
    op32 = gb.DGOperator(cells, order, precision=gb.F32,
                         kappa_cell=gb.DeviceArray.from_numpy(k[:, 0].astype(np.float32)))
    pc = gb.Preconditioner.scaled_block_jacobi(op32)
    out = []
    for chunk in (0, 16):
        u = gb.DeviceArray(op.size)
        u.clear()
        info = gb.solve_mixed(op, op32, pc, f, u, tolerance=1e-10, inner_tolerance=1e-2, max_outer=100, outer=outer,
                              graph_chunk=chunk)
        assert info.converged and info.outer_iterations > 2
        out.append((info.iterations, u.numpy()))
    (ih, uh), (ig, ug) = out
    assert abs(ig - ih) <= max(2, ih // 20)
    assert np.linalg.norm(ug - uh) <= 1e-9 * np.linalg.norm(uh)
    assert pc.status() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("cells", [(24, 24), (90, 61)])
def test_q1_general_loop(gb, cells):
    """Where the one-kernel solve cannot be placed: graph and host loop bit for bit."""
    op = gb.Q1Operator(cells, diffusion=1.0, mass=1.0)
    pc, f, out = gb.Preconditioner.diagonal(op), gb.DeviceArray.from_numpy(_rhs(cells, 2)), []
    for chunk in (0, 7):
        u = gb.DeviceArray(op.size)
        u.clear()
        rc, info = _selftest(gb, op, pc, f, u, -1, 1, 1, graph_chunk=chunk)
        assert rc == 0 and info.converged
        out.append((info.iterations, info.residual, u.numpy().tobytes()))
    assert out[0] == out[1]


@pytest.mark.gpu
@pytest.mark.parametrize("order", [3, 4])
@pytest.mark.parametrize("cells,periodic", [((5, 4, 3), (0, 0, 0)), ((20, 18, 16), (0, 1, 1)), ((40, 36, 32), (0, 0, 1))])
def test_solves_take_the_tensor_core_tiles(gb, order, cells, periodic):
    """One CG step, x = alpha P b, with the dense products on the tensor cores and in
    FP32 FMA: type changes per CTA, and on the largest grid several full tiles per CTA
    through the pipeline.  FP32 sums of up to 125 terms: the 2e-5 of the direct
    apply's test."""
    rng = np.random.default_rng(order)
    op = gb.DGOperator(cells, order, precision=gb.F32, periodic=periodic,
                       kappa_cell=gb.DeviceArray.from_numpy(rng.uniform(0.5, 2, np.prod(cells)).astype(np.float32)))
    f, out = gb.DeviceArray.from_numpy(rng.uniform(-1, 1, op.size).astype(np.float32)), {}
    for engine in ("tensor", "fma"):
        pc = gb.Preconditioner.scaled_block_jacobi(op, engine=engine)
        inv = gb.KrylovInverseOperator("cg", tolerance=1e-30, max_iterations=1)
        inv.bind(op, pc)
        for _ in range(2):
            u = gb.DeviceArray(op.size, gb.F32)
            u.clear()
            inv(f, u)
            assert pc.status() == 0
            if engine in out:  # twice the same bits
                assert np.array_equal(out[engine].view(np.uint32), u.numpy().view(np.uint32))
            out[engine] = u.numpy()
    assert np.max(np.abs(out["tensor"] - out["fma"])) <= 2e-5 * np.max(np.abs(out["fma"]))
    assert not np.array_equal(out["tensor"], out["fma"])
