"""The one-kernel FP32 closed form (dg_plane_kernel: n threads per cell, one plane
of dofs each) where its layout changes: p = 4 (bricks of 3 x 4 x 4 cells, two
spare lanes per warp) and dofs that are only 4-byte aligned, against the oracle.
The bar is the FP32 parity tests' 2e-5 of the largest entry."""
import ctypes as C

import numpy as np
import pytest

from conftest import relmax

pytestmark = pytest.mark.gpu

TOL32 = 2e-5


def _part(gb, buf, first, n):
    """n entries of a DeviceArray from `first` on, without owning them."""
    a = gb.DeviceArray.__new__(gb.DeviceArray)
    a.n, a.precision, a.itemsize = n, buf.precision, buf.itemsize
    a.free = lambda: None
    a.ptr = C.c_void_p(buf.ptr.value + first * buf.itemsize)
    return a


@pytest.mark.parametrize("cells", [(2, 2, 2), (2, 4, 5), (7, 5, 4), (10, 3, 9)])
@pytest.mark.parametrize("kw", [dict(), dict(periodic=(1, 0, 1), mass=0.7),
                                dict(diffusion=0.05, velocity=(1.0, -0.5, 0.25), periodic=(0, 1, 0))])
def test_order_four(gb, orc, cells, kw):
    prob = orc.DGProblem(cells, 4, **kw)
    u = np.random.default_rng(sum(cells)).uniform(-1, 1, prob.ndofs).astype(np.float32)
    du, w = gb.DeviceArray.from_numpy(u), gb.DeviceArray(u.size, gb.F32)
    op = gb.DGOperator(cells, 4, precision=gb.F32, **kw)
    op(du, w)
    assert relmax(w.numpy(), prob.apply(u.astype(np.float64))) < TOL32


@pytest.mark.parametrize("order", [2, 3, 4])
def test_cellwise_kappa_and_unaligned_dofs(gb, orc, order):
    cells = (9, 5, 6)
    prob = orc.DGProblem(cells, order)
    rng = np.random.default_rng(order)
    kc = np.exp(rng.uniform(-2, 2, prob.ncells))
    kfield = np.zeros(prob.ndofs)
    kfield[::(order + 1) ** 3] = kc
    u = rng.uniform(-1, 1, prob.ndofs).astype(np.float32)
    op = gb.DGOperator(cells, order, precision=gb.F32,
                       kappa_cell=gb.DeviceArray.from_numpy(kc.astype(np.float32)))
    buf = gb.DeviceArray.from_numpy(np.concatenate([[0.0], u]).astype(np.float32))
    w = gb.DeviceArray(u.size + 1, gb.F32)
    out = []
    for first_u, first_w in ((0, 0), (1, 1), (1, 0)):
        du = gb.DeviceArray.from_numpy(u) if first_u == 0 else _part(gb, buf, 1, u.size)
        dw = _part(gb, w, first_w, u.size)
        op(du, dw)
        out.append(dw.numpy().copy())
    assert np.array_equal(out[0], out[1]) and np.array_equal(out[0], out[2])
    assert relmax(out[0], prob.apply(u.astype(np.float64), kappa=kfield)) < TOL32
