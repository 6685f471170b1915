"""SSP-RK3 steps whose stages are part of the FP64 apply (full bricks and the small
ones, partial bricks, every order, with and without advection) against the same step
put together from applies.  The two differ by the roundings of the combinations:
three stages of at most three multiply-adds, each off by one unit of the sum of the
magnitudes, which the later applies (dt |L| <= 2.5 inside the stability region)
carry on: 9 (1 + 2.5 + 2.5^2) 2^-53 < 1.1e-14 of the largest term."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BOUND = 1.1e-14


@pytest.mark.parametrize("order,cells", [(1, (17, 33, 20)), (2, (33, 17, 29)), (2, (3, 2, 5)), (3, (13, 22, 19)),
                                         (3, (4, 5, 2)), (4, (17, 9, 20)), (4, (2, 3, 3))])
@pytest.mark.parametrize("kw", [dict(diffusion=0.01, velocity=(1.0, -0.5, 0.25), periodic=(1, 0, 1)),
                                dict(periodic=(0, 0, 1))])
def test_step_equals_the_step_from_applies(gb, order, cells, kw):
    op = gb.DGOperator(cells, order, **kw)
    n = cells[0] * cells[1] * cells[2] * (order + 1) ** 3
    u0 = np.random.default_rng(order + cells[0]).uniform(-1, 1, n)
    _, bound = gb.time_step_estimate(op)
    dt = 0.5 * bound
    u = gb.DeviceArray.from_numpy(u0)
    gb.RK3(op).step(u, dt)

    def apply(v):
        w = gb.DeviceArray(n)
        op(gb.DeviceArray.from_numpy(v), w)
        return w.numpy()

    f = -dt * cells[0] * cells[1] * cells[2]  # unit cube: -dt / |K|
    k0 = apply(u0)
    k1 = apply(u0 + f * k0)
    k2 = apply(u0 + 0.25 * f * k0 + 0.25 * f * k1)
    ref = u0 + f / 6 * k0 + f / 6 * k1 + 2 * f / 3 * k2
    largest = max(np.max(np.abs(u0)), *(np.max(np.abs(f * k)) for k in (k0, k1, k2)))
    assert np.max(np.abs(u.numpy() - ref)) <= BOUND * largest
