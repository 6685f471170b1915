"""The FP64 block-Jacobi apply with cell counts that leave its last CTA one cell
(the CTA's cells: 16, 7, 2 and 1 at p = 1..4) or all but one, against the dense
inverses of the operator's own blocks.  Inverting and applying in FP64 is off by
at most cond(block) nb 2^-52 of the largest entry; the blocks' condition is below 3e4
(it is computed here)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order,cells", [(1, (17, 1, 1)), (1, (3, 5, 1)), (2, (2, 2, 2)), (2, (13, 1, 1)), (2, (1, 1, 1)),
                                         (3, (3, 1, 1)), (4, (2, 1, 1))])
def test_apply_matches_the_blocks(gb, order, cells):
    op = gb.DGOperator(cells, order)
    nb, nc = (order + 1) ** 3, cells[0] * cells[1] * cells[2]
    blocks = op.block_diagonal(nb).numpy().reshape(nc, nb, nb)
    r = np.random.default_rng(order + nc).uniform(-1, 1, nc * nb)
    z = gb.DeviceArray(nc * nb)
    gb.Preconditioner.block_jacobi(op)(gb.DeviceArray.from_numpy(r), z)
    ref = np.linalg.solve(blocks, r.reshape(nc, nb, 1)).ravel()
    cond = max(np.linalg.cond(b) for b in blocks)
    assert cond < 3e4
    assert np.max(np.abs(z.numpy() - ref)) <= 2 * cond * nb * 2.0 ** -52 * np.max(np.abs(ref))
