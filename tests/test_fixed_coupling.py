"""The FP64 closed form where a line, or an entry of one, hardly enters the others: no
fewer bits than the FP64 pipe gives."""
import numpy as np
import pytest

from test_fixed_apply import apply_both, reference


@pytest.mark.gpu
@pytest.mark.parametrize("order", [1, 2, 3, 4])
@pytest.mark.parametrize("kw,step,axes", [
    (dict(diffusion=1e-6, velocity=(1.0, 0.5, 0.25)), 1e4, (0, 1, 2)),
    (dict(diffusion=1e-8, velocity=(1.0, 0.5, 0.25)), 1e6, (0, 1, 2)),
    (dict(diffusion=1e-10, velocity=(0.25, 0.5, 1.0)), 1e8, (0, 1, 2)),
    (dict(diffusion=1e-8, mass=1.0), 1e4, (0,)),  # the mass goes with the x lines
    (dict(diffusion=0.0, velocity=(1e-7, 0.0, 0.0), mass=1.0), 1e5, (0,)),
])
def test_small_coupling_to_a_large_neighbour(gb, order, kw, step, axes):
    """Cells of size 1 before cells of size `step` along one axis.  Half of the entries
    of the cells at the front are within 2^-50 of their own value: FP64 sums of some
    12 terms of about that size, typically 2^-53 each."""
    cells, n3 = (4, 4, 4), (order + 1) ** 3
    for axis in axes:
        rng = np.random.default_rng(order)
        u = rng.uniform(-1.0, 1.0, (4, 4, 4, n3))
        at = [slice(None)] * 3
        at[2 - axis] = slice(2, None)
        if kw["diffusion"] == 0.0:  # (the inflow side)
            at[2 - axis] = slice(0, 2)
        u[tuple(at)] *= step
        w = apply_both(gb, cells, order, u.ravel(), **kw)[0]
        ref = reference(cells, order, u.ravel(), **kw)[0]
        at[2 - axis] = 2 if kw["diffusion"] == 0.0 else 1
        rel = (np.abs(w - ref) / np.abs(ref)).reshape(4, 4, 4, n3)[tuple(at)]
        assert np.median(rel) <= 2.0 ** -50, axis


@pytest.mark.gpu
@pytest.mark.parametrize("order", [1, 2, 3, 4])
@pytest.mark.parametrize("cells,kw", [
    ((5, 4, 3), dict(diffusion=0.0, mass=2.0)),
    ((5, 4, 3), dict(diffusion=0.0, mass=2.0, velocity=(0.0, 0.0, 1e-30))),
    ((1, 1, 1), dict(diffusion=1e-30, mass=2.0, weak_dirichlet=False)),
])
def test_entries_of_very_different_size(gb, order, cells, kw):
    """Where the mass is all there is, every entry within 2^-52 of |K| c times its own
    coefficient (one rounding, and |K| c's), however large the others of its line are."""
    n3 = (order + 1) ** 3
    rng = np.random.default_rng(order)
    u = rng.uniform(0.5, 1.0, np.prod(cells) * n3) * 2.0 ** rng.integers(-20, 20, np.prod(cells) * n3)
    w = apply_both(gb, cells, order, u, **kw)[0]
    ref = np.float64(2.0) / np.prod(np.asarray(cells, np.longdouble)) * u
    assert np.all(np.abs(w - ref) <= 2.0 ** -51 * np.abs(ref))
