"""The FP64 apply with kappa a DG field on the integer pipes (Gauss points, block
fixed point per cell) against an extended-precision evaluation of the same
quadrature, and against the FP64-pipe kernel (which a mass of 1e-300 selects)."""
import numpy as np
import pytest

LD = np.longdouble


def legendre(n, x):
    """L_i(x), L_i'(x) of the orthonormal basis on [0,1], i < n, in extended precision: arrays [point][i]."""
    z = 2 * np.asarray(x, LD) - 1
    p, d = [np.ones_like(z), z], [np.zeros_like(z), np.ones_like(z)]
    for j in range(2, max(n, 2) + 1):
        p.append(((2 * j - 1) * z * p[-1] - (j - 1) * p[-2]) / j)
        d.append(d[-2] + (2 * j - 1) * p[j - 1])
    r = np.sqrt(2 * np.arange(n, dtype=LD) + 1)
    return np.stack(p[:n], -1) * r, 2 * np.stack(d[:n], -1) * r


def gauss(q):
    z = np.asarray(np.polynomial.legendre.leggauss(q)[0], LD)
    for _ in range(6):
        p0, p1, d0, d1 = np.ones_like(z), z, np.zeros_like(z), np.ones_like(z)
        for j in range(2, q + 1):
            p0, p1, d0, d1 = p1, ((2 * j - 1) * z * p1 - (j - 1) * p0) / j, d1, d0 + (2 * j - 1) * p1
        z = z - p1 / d1
    return (z + 1) / 2, 1 / ((1 - z * z) * d1 * d1)


def reference(cells, order, q, u, kappa, diffusion=1.0, penalty=None, weak_dirichlet=True, periodic=(0, 0, 0),
              upper=(1.0, 1.0, 1.0)):
    n = order + 1
    nx, ny, nz = cells
    eps, beta = LD(diffusion), LD(10.0 * n * n if penalty is None else penalty)
    h = [LD(upper[k]) / cells[k] for k in range(3)]
    vol = h[0] * h[1] * h[2]
    x, wt = gauss(q)
    B, G = legendre(n, x)
    V, Dv = legendre(n, np.array([0, 1], LD))
    shape = (nz, ny, nx, n, n, n)
    u, kappa = np.asarray(u, LD).reshape(shape), np.asarray(kappa, LD).reshape(shape)

    def interp(z, mats):
        for d, m in enumerate(mats):
            z = np.moveaxis(np.einsum("ij,...j->...i", m, np.moveaxis(z, 3 + d, -1)), -1, 3 + d)
        return z

    W = vol * wt[:, None, None] * wt[None, :, None] * wt[None, None, :]
    kq = interp(kappa, [B] * 3)
    w = np.zeros_like(u)
    for d in range(3):
        mats = [G if e == d else B for e in range(3)]
        w += interp(W * eps * kq * interp(u, mats), [m.T for m in mats]) / h[d] ** 2
        area, sigma, ax = vol / h[d], beta / h[d], 2 - d
        ww = (wt[:, None] * wt[None, :] * area).reshape([1 if e == d else q for e in range(3)])
        end = {}
        for s in (0, 1):
            val, slo = ([m[s:s + 1] if e == d else B for e in range(3)] for m in (V, Dv))
            end[s] = [interp(u, val), interp(u, slo) / h[d], interp(kappa, val)]
        for s in (0, 1):
            sg, sh = (1, -1) if s else (-1, 1)
            vm, dm, km = end[s]
            vp, dp, kp = (np.roll(z, sh, ax) for z in end[1 - s])
            dm, dp = sg * dm, sg * dp
            edge = np.zeros(cells[d], bool)
            if not periodic[d]:
                edge[-1 if s else 0] = True
            sp = [1] * 6
            sp[ax] = cells[d]
            edge = edge.reshape(sp)
            wd = 1 if weak_dirichlet else 0
            fv = eps * np.where(edge, wd * (sigma * km * vm - km * dm),
                                sigma * (km + kp) / 2 * (vm - vp) - (km * dm + kp * dp) / 2)
            fg = eps * np.where(edge, -wd * km * vm, -km * (vm - vp) / 2)
            w += interp(fv * ww, [V[s:s + 1].T if e == d else B.T for e in range(3)])
            w += interp(fg * ww, [sg * Dv[s:s + 1].T / h[d] if e == d else B.T for e in range(3)])
    return w.ravel()


CASES = {
    "dirichlet": dict(),
    "anisotropic": dict(upper=(1.0, 0.3, 2.0), diffusion=0.7, penalty=90.0, periodic=(0, 1, 0)),
    "no_boundary_term": dict(weak_dirichlet=False, periodic=(1, 0, 0)),
}


def fields(cells, order, seed, rough):
    nloc, nc = (order + 1) ** 3, int(np.prod(cells))
    rng = np.random.default_rng(seed)
    u = rng.uniform(-1.0, 1.0, (nc, nloc))
    k = np.zeros((nc, nloc))
    k[:, 0] = np.exp(rng.normal(0.0, 1.0, nc))
    k[:, 1:] = 0.02 * k[:, :1] * rng.uniform(-1.0, 1.0, (nc, nloc - 1))
    if rough:  # magnitudes of their own in every cell; a smooth part that dwarfs the rest
        u[:, 0] += 50.0
        u *= 2.0 ** rng.integers(-20, 20, (nc, 1))
        k *= 2.0 ** rng.integers(-20, 20, (nc, 1))
    return u.ravel(), k.ravel()


def apply_both(gb, cells, order, q, u, k, **kw):
    out = []
    ud, kd = gb.DeviceArray.from_numpy(u), gb.DeviceArray.from_numpy(k)
    for mass in (0.0, 1e-300):
        op = gb.DGOperator(cells, order, quad_points=q, kappa=kd, mass=mass, **kw)
        w = gb.DeviceArray(op.size)
        op(ud, w)
        out.append(w.numpy())
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("order", [1, 2, 3, 4])
@pytest.mark.parametrize("extra", [1, 2])
@pytest.mark.parametrize("case", sorted(CASES))
@pytest.mark.parametrize("rough", [False, True])
def test_error_is_no_larger_than_the_fp64_kernels(gb, order, extra, case, rough):
    """Within 1e-12 in the max norm (the framework's bound for FP64), and, over the
    cells relative to each cell's largest entry, a root mean square error no
    larger than that of the FP64-pipe kernel."""
    kw, q = CASES[case], order + extra
    for cells in ((2, 3, 2), (9, 5, 3)):
        u, k = fields(cells, order, 10 * order + extra, rough)
        w, w2 = apply_both(gb, cells, order, q, u, k, **kw)
        ref = reference(cells, order, q, u, k, **kw)
        assert np.max(np.abs(w - ref)) <= 1e-12 * np.max(np.abs(ref))
        big = np.max(np.abs(ref.reshape(np.prod(cells), -1)), axis=1, keepdims=True)
        err, err2 = (np.abs(v - ref).reshape(big.size, -1) / big for v in (w, w2))
        assert np.sqrt(np.mean(err ** 2)) <= np.sqrt(np.mean(err2 ** 2)), cells


@pytest.mark.gpu
@pytest.mark.parametrize("order", [1, 3, 4])
def test_values_beyond_the_fixed_point_range(gb, order):
    """Zeros, subnormals, the ends of the range, infinities, NaN in u and in
    kappa: the entries of the FP64-pipe kernel, non-finite where it is, bit for
    bit in the cells next to them."""
    cells = (7, 5, 6)
    nloc = (order + 1) ** 3
    for where in ("u", "kappa"):
        for mark in (0.0, 5e-324, 1e-260, 1e200, np.inf, np.nan):
            u, k = fields(cells, order, order, False)
            (u if where == "u" else k)[100 * nloc:101 * nloc] *= mark if np.isfinite(mark) else 1.0
            (u if where == "u" else k)[100 * nloc + 3] = mark
            w, w2 = apply_both(gb, cells, order, 0, u, k)
            assert np.array_equal(np.isfinite(w), np.isfinite(w2)), (where, mark)
            a, b = w.reshape(-1, nloc)[100], w2.reshape(-1, nloc)[100]
            fine = np.isfinite(b)
            assert np.all(np.abs(a - b)[fine] <= 1e-12 * max(np.max(np.abs(b[fine]), initial=0.0), 1e-300)), (where, mark)
    u, k = fields(cells, order, order, False)
    w, _ = apply_both(gb, cells, order, 0, 0 * u, k)
    assert not w.any()


@pytest.mark.gpu
@pytest.mark.parametrize("order", [1, 2, 3, 4])
def test_zero_at_the_ends_of_the_scales(gb, order):
    """u = 0 gives 0 where operator and kappa are as small as fixed point takes them."""
    cells, n3 = (2, 2, 3), (order + 1) ** 3
    k = np.zeros((12, n3))
    u, w = gb.DeviceArray(12 * n3), gb.DeviceArray(12 * n3)
    u.clear()
    for e in range(80, 101):
        k[:, 0] = 2.0 ** -e
        for eps in (2.0 ** -100, 2.0 ** -102, 2.0 ** -104, 2.0 ** -106, 2.0 ** -108):
            op = gb.DGOperator(cells, order, kappa=gb.DeviceArray.from_numpy(k.ravel()), diffusion=eps)
            op(u, w)
            assert not w.numpy().any(), (e, eps)


@pytest.mark.gpu
@pytest.mark.parametrize("order", [1, 2, 3, 4])
def test_without_memory_for_the_tables(gb, order):
    """The operator is made all the same and gives the FP64 kernel's bits, also after
    an update of kappa."""
    cells, n3 = (5, 4, 3), (order + 1) ** 3
    rng = np.random.default_rng(order)
    k = np.zeros((60, n3))
    k[:, 0], k[:, 1] = rng.uniform(1.0, 2.0, 60), rng.uniform(-0.2, 0.2, 60)
    kappa = gb.DeviceArray.from_numpy(k.ravel())
    u = gb.DeviceArray.from_numpy(rng.uniform(-1.0, 1.0, 60 * n3))
    ref, w = gb.DeviceArray(60 * n3), gb.DeviceArray(60 * n3)
    gb.DGOperator(cells, order, kappa=kappa, mass=1e-300)(u, ref)
    gb.check(gb.lib().gbfem_selftest_no_fixed_memory(1))
    try:
        op = gb.DGOperator(cells, order, kappa=kappa)
    finally:
        gb.check(gb.lib().gbfem_selftest_no_fixed_memory(0))
    op(u, w)
    assert np.array_equal(w.numpy(), ref.numpy())
    gb.check(gb.lib().gbfem_operator_update_coefficients(op.handle))
    op(u, w)
    assert np.array_equal(w.numpy(), ref.numpy())
