"""The scaled shared-block Jacobi in its tensor-product form (fast
diagonalisation) against dense FP64 inverses of the oracle's kappa = 1 blocks."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("order", [1, 2, 3, 4])
@pytest.mark.parametrize("cells,kw", [
    ((1, 1, 1), dict()),                                     # both boundaries on every axis, less than one warp of cells
    ((2, 1, 7), dict(upper=(1.0, 0.3, 2.0), diffusion=2.5)),  # no interior cell, anisotropic
    ((9, 6, 5), dict(upper=(1.0, 0.25, 3.0), penalty=55.0)),
    ((33, 4, 3), dict(periodic=(0, 1, 0))),                  # CTAs with and without boundary cells
])
def test_against_dense_inverse(gb, orc, order, cells, kw):
    """Relative to the largest entry of each cell's result: FP32 rounding of r
    in the eigenbasis (2^-24 a step, about 6 n steps of sums) divided by the
    smallest eigenvalue, against |z| >= |r| / (largest eigenvalue) -- bounded
    here by the blocks' own condition number: 40 2^-24 cond."""
    nc, nloc = int(np.prod(cells)), (order + 1) ** 3
    rng = np.random.default_rng(order)
    kc = np.exp(rng.uniform(-2, 2, nc)).astype(np.float32)
    r = rng.uniform(-1, 1, nc * nloc).astype(np.float32)
    op = gb.DGOperator(cells, order, precision=gb.F32, kappa_cell=gb.DeviceArray.from_numpy(kc), **kw)
    z = gb.DeviceArray(nc * nloc, gb.F32)
    gb.Preconditioner.scaled_block_jacobi(op)(gb.DeviceArray.from_numpy(r), z)
    blocks = orc.DGProblem(cells, order, **kw).block_diagonal(nthreads=4)
    ref = np.linalg.solve(blocks, r.astype(np.float64).reshape(nc, nloc, 1))[..., 0] / kc[:, None]
    err = np.max(np.abs(z.numpy().reshape(nc, nloc) - ref), axis=1) / np.max(np.abs(ref), axis=1)
    assert np.all(err <= 40 * 2.0 ** -24 * np.linalg.cond(blocks))
    assert np.sqrt(np.mean(err ** 2)) < 2e-5


@pytest.mark.gpu
@pytest.mark.parametrize("engine", ["tensor", "fma"])
def test_singular_blocks_are_refused(gb, engine):
    """No diffusion: the blocks are zero."""
    op = gb.DGOperator((3, 2, 1), 2, precision=gb.F32, diffusion=0.0,
                       kappa_cell=gb.DeviceArray.from_numpy(np.ones(6, np.float32)))
    with pytest.raises(gb.GbfemError):
        gb.Preconditioner.scaled_block_jacobi(op, engine=engine)


@pytest.mark.gpu
@pytest.mark.parametrize("order", [1, 2])
def test_block_singular_up_to_rounding(gb, order):
    """One cell whose constants nothing holds: the dense inverse of the rounded
    block, with either engine."""
    op = gb.DGOperator((1, 1, 1), order, precision=gb.F32, weak_dirichlet=False,
                       kappa_cell=gb.DeviceArray.from_numpy(np.ones(1, np.float32)))
    r = gb.DeviceArray.from_numpy(np.random.default_rng(1).uniform(-1, 1, op.size).astype(np.float32))
    out = []
    for engine in ("tensor", "fma"):
        z = gb.DeviceArray(op.size, gb.F32)
        try:
            gb.Preconditioner.scaled_block_jacobi(op, engine=engine)(r, z)
            out.append(z.numpy().view(np.uint32).tolist())
        except gb.GbfemError as e:
            out.append(str(e))
    assert out[0] == out[1]


@pytest.mark.gpu
@pytest.mark.parametrize("order", [1, 2])
def test_low_orders_keep_the_dense_products(gb, order):
    """p <= 2: sums of at most 27 FP32 products, which the diagonalised form's six
    rounded contractions do not match: the dense engine's bits."""
    cells = (11, 10, 9)
    rng = np.random.default_rng(order)
    op = gb.DGOperator(cells, order, precision=gb.F32,
                       kappa_cell=gb.DeviceArray.from_numpy(np.exp(rng.uniform(-2, 2, 990)).astype(np.float32)))
    r = gb.DeviceArray.from_numpy(rng.uniform(-1, 1, op.size).astype(np.float32))
    out = []
    for engine in ("tensor", "fma"):
        z = gb.DeviceArray(op.size, gb.F32)
        gb.Preconditioner.scaled_block_jacobi(op, engine=engine)(r, z)
        out.append(z.numpy())
    assert np.array_equal(*out)


@pytest.mark.gpu
@pytest.mark.parametrize("order", [3, 4])
@pytest.mark.parametrize("kw,dense", [(dict(), False), (dict(penalty=0.3), True), (dict(penalty=1.0), True),
                                      (dict(penalty=1.0, weak_dirichlet=False, upper=(1.0, 0.5, 2.0)), True)])
def test_indefinite_blocks_take_the_dense_products(gb, order, kw, dense):
    """A small penalty: the sums of the 1-D eigenvalues cancel, and the division would
    amplify their rounding.  The direct apply z = P r is then the solves': the first
    CG iterate is alpha z, rounded once, for one FP32 alpha."""
    cells, n = (6, 7, 3), 126 * (order + 1) ** 3
    rng = np.random.default_rng(order)
    op = gb.DGOperator(cells, order, precision=gb.F32,
                       kappa_cell=gb.DeviceArray.from_numpy(np.exp(rng.uniform(-1, 1, 126)).astype(np.float32)), **kw)
    pc = gb.Preconditioner.scaled_block_jacobi(op)
    inv = gb.KrylovInverseOperator("cg", tolerance=1e-30, max_iterations=1)
    inv.bind(op, pc)
    for _ in range(40):  # <r, P r> > 0, or there is no step
        r, z, x = gb.DeviceArray.from_numpy(rng.uniform(-1, 1, n).astype(np.float32)), *(gb.DeviceArray(n, gb.F32) for _ in "zx")
        x.clear()
        inv(r, x)
        if x.numpy().any():
            break
    pc(r, z)
    x, z = x.numpy(), z.numpy()
    j = np.argmax(np.abs(x))
    near = [np.float32(x[j] / z[j])]
    for way in (np.float32(-np.inf), np.float32(np.inf)):
        near += [np.nextafter(near[0], way), np.nextafter(np.nextafter(near[0], way), way)]
    assert x.any() and any(np.array_equal(a * z, x) for a in near) == dense
