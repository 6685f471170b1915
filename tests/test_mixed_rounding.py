"""The mixed solve keeps its rounding.

The inner FP32 CG amplifies every rounding of its residual, its preconditioner
and the FP64 product that forms the residual.  Where the outer iteration does
not converge (kappa negative at points: the operator is indefinite) its result
is one particular iterate, and another rounding gives another one, 1e-5 to 1e-3
away.  The values below were computed with the outer product on the FP64 pipe and
the preconditioner as products with the dense inverses; all inputs are dyadic
numbers of integer arithmetic, the same on every machine."""
import numpy as np
import pytest

CELLS = (6, 7, 8)


def _dyadic(n, salt):
    """n values in (-1, 1), multiples of 2^-20 (SplitMix64)."""
    with np.errstate(over="ignore"):
        z = np.uint64(salt) + np.uint64(0x9E3779B97F4A7C15) * np.arange(1, n + 1, dtype=np.uint64)
        z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
    z ^= z >> np.uint64(31)
    return (z >> np.uint64(43)).astype(np.float64) * 2.0 ** -20 - 1.0


def solve(gb, order, engine, cells=CELLS):
    nc, nloc = int(np.prod(cells)), (order + 1) ** 3
    k = _dyadic(nc * nloc, 7 + order).reshape(nc, nloc) * 0.25
    k[:, 0] = 1.0 + 0.5 * _dyadic(nc, 1)
    f = np.zeros((nc, nloc))
    f[:, 0] = 2.0 ** -9 * (1.0 + 0.5 * _dyadic(nc, 2))
    op = gb.DGOperator(cells, order, kappa=gb.DeviceArray.from_numpy(k.ravel()))
    op32 = gb.DGOperator(cells, order, precision=gb.F32,
                         kappa_cell=gb.DeviceArray.from_numpy(k[:, 0].astype(np.float32)))
    pc = gb.Preconditioner.scaled_block_jacobi(op32, engine=engine)
    u = gb.DeviceArray(op.size)
    u.clear()
    info = gb.solve_mixed(op, op32, pc, gb.DeviceArray.from_numpy(f.ravel()), u, tolerance=1e-10, inner_tolerance=1e-2,
                          max_outer=40, outer="fgmres", outer_restart=10, graph_chunk=16)
    return info, u.numpy()


# (order, engine): entries 0, s, 2 s, ... of the result, s a sixth of its size
RESULTS = {
    (1, 'fma'): ('0x1.1cfde259cd703p-10', '0x1.6b5f48101ea50p-6', '0x1.7b22e26f2d962p-6',
                 '0x1.da7fa6aed70ccp-9', '0x1.ddf9f796fc29bp-6', '0x1.1d91e2032894ep-6'),
    (2, 'fma'): ('0x1.bfff2273b1f7fp-13', '0x1.89f9d282c42e1p-9', '0x1.924f712e77133p-9',
                 '0x1.3c10e398bad45p-11', '0x1.04b9272406b71p-8', '0x1.44fa855d33086p-9'),
    (3, 'fma'): ('0x1.de8c54ef3d7e3p-16', '0x1.a1ecb976dbeb9p-12', '0x1.ab1c48ec389abp-12',
                 '0x1.5b3882d92c508p-14', '0x1.137754a337aa6p-11', '0x1.5c9e656252120p-12'),
    (4, 'fma'): ('0x1.5530a600e4d65p-18', '0x1.1a135edcfd48fp-14', '0x1.1ebaa6c76530fp-14',
                 '0x1.cd71a4c410e2ep-17', '0x1.794e3e440c769p-14', '0x1.cf3085266557cp-15'),
    (1, 'tensor'): ('0x1.1cfde259cd703p-10', '0x1.6b5f48101ea50p-6', '0x1.7b22e26f2d962p-6',
                 '0x1.da7fa6aed70ccp-9', '0x1.ddf9f796fc29bp-6', '0x1.1d91e2032894ep-6'),
    (2, 'tensor'): ('0x1.bfff2273b1f7fp-13', '0x1.89f9d282c42e1p-9', '0x1.924f712e77133p-9',
                 '0x1.3c10e398bad45p-11', '0x1.04b9272406b71p-8', '0x1.44fa855d33086p-9'),
    (3, 'tensor'): ('0x1.de8a3a246218bp-16', '0x1.a1ebeaa51e4b7p-12', '0x1.ab1b95caaa7dbp-12',
                 '0x1.5b3797e6aeb1ep-14', '0x1.1376ea3cda877p-11', '0x1.5c9d548090448p-12'),
    (4, 'tensor'): ('0x1.55318d36c9b72p-18', '0x1.1a143ab635676p-14', '0x1.1ebb9de7475a4p-14',
                 '0x1.cd731c499a874p-17', '0x1.794f779f4e6c1p-14', '0x1.cf31d8375a080p-15'),
}


@pytest.mark.gpu
@pytest.mark.parametrize("order,engine", sorted(RESULTS))
def test_result_of_a_stagnating_solve(gb, order, engine):
    """Within 1e-9 of the recorded entries, relative to the largest of them."""
    info, u = solve(gb, order, engine)
    ref = np.array([float.fromhex(v) for v in RESULTS[order, engine]])
    assert not info.converged and info.stagnated
    assert np.max(np.abs(u[::u.size // 6][:6] - ref)) <= 1e-9 * np.max(np.abs(ref))
