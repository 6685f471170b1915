"""The FP64 closed form on the integer pipes (one kernel, block fixed point per
line) against an extended-precision evaluation of the same formulas, and
against the FP64-pipe kernels over every input both accept."""
import ctypes as C

import numpy as np
import pytest

LD = np.longdouble


def legendre_ends(n):
    """L_i(s), L_i'(s) of the orthonormal basis on [0,1] at s = 0, 1."""
    i = np.arange(n)
    r = np.sqrt(LD(2) * i + 1)
    v = np.array([r * LD(-1) ** i, r])
    d = r * i * (i + 1)
    return v, np.array([d * LD(-1) ** (i + 1), d])


def line_matrices(n):
    """K1 = int L_i' L_j', D1 = int L_i' L_j, from L_i' = sum of 2 r_i r_k L_k over k < i, i + k odd."""
    r = np.sqrt(LD(2) * np.arange(n) + 1)
    D = np.zeros((n, n), LD)
    for i in range(n):
        for k in range(i):
            if (i + k) % 2:
                D[i, k] = 2 * r[i] * r[k]
    return D @ D.T, D


def reference(cells, order, u, diffusion=1.0, penalty=None, mass=0.0, velocity=(0, 0, 0), weak_dirichlet=True,
              periodic=(0, 0, 0), upper=(1.0, 1.0, 1.0)):
    """(w, s): A u in extended precision, and the sum of the absolute values of
    the terms of every entry (with the largest coefficient of each line in the
    place of all of them): the size that rounding errors are relative to."""
    n = order + 1
    nx, ny, nz = cells
    eps, beta = LD(diffusion), LD(10.0 * n * n if penalty is None else penalty)
    h = [LD(upper[k]) / cells[k] for k in range(3)]
    vol = h[0] * h[1] * h[2]
    V, Dv = legendre_ends(n)
    K1, D1 = line_matrices(n)
    x = np.asarray(u, LD).reshape(nz, ny, nx, n, n, n)
    w, size = np.zeros_like(x), np.zeros_like(x)
    for d in range(3):
        a, b = 3 + d, LD(velocity[d])
        big = np.abs(np.broadcast_to(np.max(np.abs(x), axis=a, keepdims=True), x.shape))

        def along(m, z):
            # m applied along local axis a (einsum has no BLAS path for extended precision)
            return np.moveaxis(np.einsum("ij,...j->...i", m, np.moveaxis(z, a, -1)), -1, a)

        M = eps * vol / h[d] ** 2 * K1 - b * vol / h[d] * D1 + (LD(mass) * vol * np.eye(n, dtype=LD) if d == 0 else 0)
        w += along(M, x)
        size += along(np.abs(M), big)
        area, A2 = vol / h[d], vol / h[d] * eps / (2 * h[d])
        A1 = area * eps * beta / h[d]
        for s in (0, 1):
            ax, sh, sg = 2 - d, (-1 if s else 1), (1 if s else -1)
            v, g = along(V[s:s + 1], x), sg * along(Dv[s:s + 1], x)
            vn, gn = (np.roll(along(t[1 - s:2 - s], x), sh, ax) for t in (V, Dv))
            gn = sg * gn
            S, G = along(np.abs(V[s:s + 1]), big), along(np.abs(Dv[s:s + 1]), big)
            Sn, Gn = np.roll(S, sh, ax), np.roll(G, sh, ax)
            bn = area * b * sg
            val = A1 * (v - vn) - A2 * (g + gn) + bn * (v if bn >= 0 else vn)
            gr = -A2 * (v - vn)
            sval = A1 * (S + Sn) + A2 * (G + Gn) + abs(bn) * (S + Sn)
            sgr = A2 * (S + Sn)
            edge = np.zeros(cells[d], bool)
            if not periodic[d]:
                edge[-1 if s else 0] = True
            shape = [1] * 6
            shape[ax] = cells[d]
            edge = edge.reshape(shape)
            wd = 1 if weak_dirichlet else 0
            val = np.where(edge, wd * (A1 * v - 2 * A2 * g) + max(bn, LD(0)) * v, val)
            gr = np.where(edge, wd * (-2 * A2 * v), gr)
            sval = np.where(edge, A1 * S + 2 * A2 * G + abs(bn) * S, sval)
            sgr = np.where(edge, 2 * A2 * S, sgr)
            w += along(V[s:s + 1].T, val) + along((sg * Dv[s:s + 1]).T, gr)
            size += along(np.abs(V[s:s + 1]).T, sval) + along(np.abs(Dv[s:s + 1]).T, sgr)
    return w.ravel(), size.ravel()


CASES = {
    "poisson": dict(),
    "advection_mass": dict(diffusion=0.03, velocity=(1.0, -0.5, 0.25), mass=2.0),
    "periodic_advection": dict(diffusion=1e-3, velocity=(-1.0, 0.5, 0.0), periodic=(1, 1, 1), weak_dirichlet=False),
    "no_boundary_term": dict(weak_dirichlet=False, periodic=(0, 1, 0), mass=1.0),
    "no_penalty": dict(penalty=0.0, upper=(1.0, 0.5, 2.0)),
    "pure_advection": dict(diffusion=0.0, velocity=(1.0, -0.5, 0.25), periodic=(0, 0, 1)),
}
# one brick or less, ragged bricks in each direction, several bricks
GRIDS = [(1, 1, 1), (2, 3, 2), (9, 5, 3), (5, 9, 6), (17, 4, 5)]


def apply_both(gb, cells, order, u, **kw):
    """(integer-pipe result, FP64-pipe result): the second from the closed form
    with kappa = 1 given per cell, with advection from the Gauss points."""
    ud = gb.DeviceArray.from_numpy(u)
    if "velocity" in kw:
        other = gb.DGOperator(cells, order, algorithm=gb.ALGO_QUADRATURE, **kw)
    else:
        other = gb.DGOperator(cells, order, kappa_cell=gb.DeviceArray.from_numpy(np.ones(np.prod(cells))), **kw)
    out = []
    for op in (gb.DGOperator(cells, order, **kw), other):
        w = gb.DeviceArray(op.size)
        op(ud, w)
        out.append(w.numpy())
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("order", [1, 2, 3, 4])
@pytest.mark.parametrize("case", sorted(CASES))
def test_entrywise_error_and_no_worse_than_fp64(gb, order, case):
    """Every entry within 2^-49 of the size of its terms: a trace unit is 2^-55
    of its line's largest coefficient, a face difference holds at most four,
    and two faces of two traces, the row's own rounding (2^-54) and the FP64
    sum over the axes stay below 2^-49.  Over all entries the error is no larger
    than that of the FP64 kernels."""
    kw = CASES[case]
    for k, cells in enumerate(GRIDS):
        if any(p and c < 2 for p, c in zip(kw.get("periodic", (0, 0, 0)), cells)):
            continue
        n3 = (order + 1) ** 3
        rng = np.random.default_rng(100 * order + k)
        u = rng.uniform(-1.0, 1.0, np.prod(cells) * n3)
        if k % 2:  # magnitudes of their own in every cell and mode
            u *= 2.0 ** rng.integers(-30, 30, np.prod(cells)).repeat(n3) * 2.0 ** rng.integers(-20, 20, u.size)
        w, w2 = apply_both(gb, cells, order, u, **kw)
        ref, size = reference(cells, order, u, **kw)
        err, err2 = (np.abs(v - ref) / size for v in (w, w2))
        assert np.all(err <= 2.0 ** -49), (cells, float(err.max()))
        if cells != (1, 1, 1):
            assert np.sqrt(np.mean(err ** 2)) <= np.sqrt(np.mean(err2 ** 2)), cells


@pytest.mark.gpu
@pytest.mark.parametrize("order", [1, 2, 3, 4])
@pytest.mark.parametrize("case", ["poisson", "advection_mass", "no_boundary_term"])
def test_magnitudes_and_special_values(gb, order, case):
    """Zeros, the ends of the FP64 range, subnormals, infinities and NaN:
    non-finite in the lines of a non-finite entry and of its neighbours, as the
    FP64 closed form is, the others within 2^-48 of their terms (2^-49, and the
    FP64 lines' own rounding)."""
    kw, cells = CASES[case], (5, 4, 6)
    plain = {k: v for k, v in kw.items() if k != "velocity"}
    n3 = (order + 1) ** 3
    rng = np.random.default_rng(order)
    base = rng.uniform(-1.0, 1.0, (np.prod(cells), n3))
    for mark in (0.0, 1e-300, 1e280, 5e-324, np.inf, -np.inf, np.nan):
        u = base.copy()
        u[7] *= mark if np.isfinite(mark) else 1.0
        u[60, 3] = mark
        u[61] = 0.0
        u[62] *= 1e-290
        u = u.ravel()
        w = apply_both(gb, cells, order, u, **kw)[0]
        assert np.array_equal(np.isfinite(w), np.isfinite(apply_both(gb, cells, order, u, **plain)[1])), mark
        with np.errstate(invalid="ignore"):
            ref, size = reference(cells, order, u, **kw)
            fine = np.isfinite(w) & np.isfinite(ref.astype(float))
            # a subnormal spacing covers what underflows
            assert np.all(np.abs(w - ref)[fine] <= 2.0 ** -48 * size[fine] + 64 * 5e-324), mark
    u = np.zeros(np.prod(cells) * n3)
    w, _ = apply_both(gb, cells, order, u, **kw)
    assert not w.any()


@pytest.mark.gpu
@pytest.mark.parametrize("order", [1, 2, 3, 4])
def test_constant_is_in_the_kernel_and_odd_addresses(gb, order):
    """A constant gives exactly zero without a boundary term; vectors that
    start at an odd multiple of 8 bytes give the same bits."""
    cells, n3 = (6, 5, 7), (order + 1) ** 3
    n = np.prod(cells) * n3
    u = np.zeros((np.prod(cells), n3))
    u[:, 0] = 0.1
    op = gb.DGOperator(cells, order, weak_dirichlet=False, periodic=(1, 0, 1))
    w = gb.DeviceArray(n)
    op(gb.DeviceArray.from_numpy(u.ravel()), w)
    assert not w.numpy().any()
    v = np.random.default_rng(order).uniform(-1.0, 1.0, n)
    op(gb.DeviceArray.from_numpy(v), w)
    pad = gb.DeviceArray.from_numpy(np.concatenate([[7.0], v]))
    out = gb.DeviceArray(n + 1)
    gb.check(gb.lib().gbfem_operator_apply(op.handle, C.c_void_p(pad.ptr.value + 8), C.c_void_p(out.ptr.value + 8),
                                           None))
    assert np.array_equal(out.numpy()[1:], w.numpy())


@pytest.mark.gpu
def test_refused_coefficients_take_the_fp64_kernels(gb):
    """A penalty so small that P = v - r dv outgrows v."""
    cells, u = (5, 4, 3), np.random.default_rng(3).uniform(-1.0, 1.0, 5 * 4 * 3 * 64)
    w, w2 = apply_both(gb, cells, 3, u, penalty=1e-3)
    assert np.max(np.abs(w - w2)) <= 1e-12 * np.max(np.abs(w2))


@pytest.mark.gpu
@pytest.mark.parametrize("order", [1, 2, 3, 4])
@pytest.mark.parametrize("velocity", [(1.0, -0.5, 0.25), (1.0, 0.0, 0.0)])
def test_extreme_lines_beside_uncoupled_neighbours(gb, order, velocity):
    """Without diffusion an outflow neighbour, or any neighbour along an axis
    without velocity, has no part in a line: lines that fixed point cannot hold
    beside ordinary ones, each within 2^-48 of its own terms."""
    kw, cells = dict(diffusion=0.0, velocity=velocity), (5, 4, 6)
    n3 = (order + 1) ** 3
    base = np.random.default_rng(order).uniform(-1.0, 1.0, (np.prod(cells), n3))
    for mark in (1e-250, 1e-300, 1e280):
        u = base.copy()
        u[[7, 60, 61, 93]] *= mark
        u = u.ravel()
        w = apply_both(gb, cells, order, u, **kw)[0]
        ref, size = reference(cells, order, u, **kw)
        assert np.all(np.abs(w - ref) <= 2.0 ** -48 * size + 64 * 5e-324), mark


@pytest.mark.gpu
@pytest.mark.parametrize("kw", [dict(mass=np.nan), dict(velocity=(0.5, np.nan, 0.0)), dict(velocity=(0.5, np.inf, 0.0)),
                                dict(diffusion=np.nan), dict(penalty=np.nan)])
def test_non_finite_coefficients(gb, kw):
    """The result is not finite either."""
    op = gb.DGOperator((3, 4, 2), 2, **kw)
    w = gb.DeviceArray(op.size)
    op(gb.DeviceArray.from_numpy(np.random.default_rng(1).uniform(0.5, 1.0, op.size)), w)
    assert not np.any(np.isfinite(w.numpy().reshape(-1, 27)[:, 0]))
