"""The FP64 reaction term on the integer pipes: its exp on the host, and the
kernels against an extended-precision evaluation of the same quadrature."""
import ctypes as C

import numpy as np
import pytest

from test_quad_fixed import LD, gauss, legendre


def test_exp_against_extended_precision(gb):
    """0.52 units in the last place up to |x| = 64 and 0.65 up to 700 (half from
    the final rounding; 64-bit log2(e) contributes |x| 2^-64, the truncations
    below 2^-60); the special values are the C library's."""
    f = gb.lib().gbfem_selftest_exp
    f.argtypes = [C.c_int64, C.c_void_p, C.c_void_p]
    rng = np.random.default_rng(1)
    for scale, bound in ((1e-300, 0.5), (1e-17, 0.51), (1e-8, 0.52), (1e-3, 0.52), (1.0, 0.52), (64.0, 0.52), (699.0, 0.65)):
        x = np.concatenate([rng.uniform(-scale, scale, 50000), [scale, -scale, scale / 3]])
        y = np.empty_like(x)
        assert f(x.size, x.ctypes.data, y.ctypes.data) == 0
        ref = np.exp(x.astype(LD))
        assert np.max(np.abs(y - ref) / np.spacing(ref.astype(float))) <= bound, scale
    # steps of the table and multiples of ln 2
    x = np.concatenate([np.arange(-700, 700) * np.log(2) / 32, np.arange(-1000, 1000) * np.log(2)])
    y = np.empty_like(x)
    f(x.size, x.ctypes.data, y.ctypes.data)
    assert np.max(np.abs(y / np.exp(x.astype(LD)) - 1)) < 2.0 ** -52
    x = np.array([0.0, -0.0, 5e-324, -5e-324, 710.0, -746.0, np.inf, -np.inf, np.nan])
    y = np.empty_like(x)
    f(x.size, x.ctypes.data, y.ctypes.data)
    assert np.array_equal(y, np.array([1.0, 1.0, 1.0, 1.0, np.inf, 0.0, np.inf, 0.0, np.nan]), equal_nan=True)


def parts(cells, order, extra):
    n, q = order + 1, order + extra
    x, wt = gauss(q)
    B = legendre(n, x)[0]
    W = wt[:, None, None] * wt[None, :, None] * wt[None, None, :] / np.prod(cells)

    def along(z, m):
        for d in range(3):
            z = np.moveaxis(np.einsum("ij,...j->...i", m, np.moveaxis(z, 1 + d, -1)), -1, 1 + d)
        return z

    return n, B, W, along


EXPR = {(0.0, 0.0, -5.0): "-5.0 * exp(u)", (1.5, -0.25, 0.0): "1.5 * u - 0.25 * u * u * u",
        (0.5, 2.0, 0.1): "0.5 * u + 2.0 * u * u * u + 0.1 * exp(u)"}


@pytest.mark.gpu
@pytest.mark.parametrize("order", [1, 2, 3, 4])
@pytest.mark.parametrize("extra", [1, 2])
@pytest.mark.parametrize("reaction", sorted(EXPR))
def test_reaction_and_its_linearisation(gb, order, extra, reaction):
    """R(u) and R'(u) d alone (an operator without a linear part): within 1e-12 in
    the max norm, and R(u), relative to each cell's largest entry, with a root
    mean square error no larger than that of the FP64-pipe kernel, which the same
    reaction as a user's expression still takes."""
    import integrands
    c1, c3, ce = reaction
    for cells in ((1, 1, 1), (3, 5, 7)):
        n, B, W, along = parts(cells, order, extra)
        nc = int(np.prod(cells))
        rng = np.random.default_rng(order)
        u, d = rng.uniform(-0.6, 0.6, (nc, n, n, n)), rng.uniform(-1.0, 1.0, (nc, n, n, n))
        u[nc // 2] = 0.0
        kw = dict(quad_points=order + extra, diffusion=0.0)
        op = gb.NonlinearDGOperator(cells, order, reaction=reaction, **kw)
        user = integrands.UserNonlinearDGOperator(cells, order, EXPR[reaction], **kw)
        ud, w, w2, z = (gb.DeviceArray.from_numpy(u.ravel()), *(gb.DeviceArray(u.size) for _ in range(3)))
        op(ud, w)
        user(ud, w2)
        op.jacobian(ud)(gb.DeviceArray.from_numpy(d.ravel()), z)
        uq, dq = along(u.astype(LD), B), along(d.astype(LD), B)
        ref = along(W * (c1 * uq + c3 * uq ** 3 + ce * np.exp(uq)), B.T)
        lin = along(W * (c1 + 3 * c3 * uq ** 2 + ce * np.exp(uq)) * dq, B.T)
        w, w2, z = (v.numpy().reshape(ref.shape) for v in (w, w2, z))
        assert np.max(np.abs(w - ref)) <= 1e-12 * np.max(np.abs(ref))
        assert np.max(np.abs(z - lin)) <= 1e-12 * np.max(np.abs(lin))
        if nc > 1:
            big = np.max(np.abs(ref), axis=(1, 2, 3), keepdims=True)
            big[big == 0] = 1
            err, err2 = (np.abs(v - ref) / big for v in (w, w2))
            assert np.sqrt(np.mean(err ** 2)) <= np.sqrt(np.mean(err2 ** 2))


@pytest.mark.gpu
def test_values_beyond_the_range(gb):
    """An infinity, a NaN, an overflow of exp and the ends of the range: nothing
    beyond the cells that hold them is affected (and their face neighbours, whose
    jumps, times a diffusion of zero, are the linear part's)."""
    cells, order = (5, 4, 3), 2
    rng = np.random.default_rng(3)
    u = rng.uniform(-0.5, 0.5, (60, 27))
    op = gb.NonlinearDGOperator(cells, order, reaction=(0.0, 1.0, 1.0), diffusion=0.0)
    w = gb.DeviceArray(u.size)
    op(gb.DeviceArray.from_numpy(u.ravel()), w)
    plain = w.numpy().reshape(60, 27)
    for mark, finite in ((np.inf, False), (np.nan, False), (2000.0, False), (1e-250, True), (5e-324, True)):
        v = u.copy()
        v[17] = 0.0
        v[17, 0] = mark
        op(gb.DeviceArray.from_numpy(v.ravel()), w)
        got = w.numpy().reshape(60, 27)
        x, y, z = (v - o for v, o in zip(np.unravel_index(np.arange(60), (3, 4, 5))[::-1], (2, 3, 0)))  # 17 is (2, 3, 0)
        rest = np.abs(x) + np.abs(y) + np.abs(z) > 1
        assert np.max(np.abs(got[rest] - plain[rest])) <= 1e-15 * np.max(np.abs(plain)), mark
        assert bool(np.all(np.isfinite(got[17]))) == finite, mark
        if finite:  # r = e^0 = 1: the load vector of 1
            assert abs(got[17, 0] - 1.0 / 60) < 1e-16 and np.max(np.abs(got[17, 1:])) < 1e-17, mark
