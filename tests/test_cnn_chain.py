"""The learned preconditioner's forward pass as a chain of overlapping kernels:
grids whose levels take the convolution of few positions (16 per CTA, ragged ends:
20^3 to 3^3), against the oracle in arithmetic that is exact in FP32, and passes and
training steps issued back to back against the same ones with a wait in between."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [16, 24, 40])
def test_small_grid_convolutions_are_exact(gb, N):
    """One tap per 3x3x3 layer, a scaled permutation as its channel matrix, weights
    in {1/2, 1, 2}, inputs +-1: every sum is exact, so the outputs agree bitwise."""
    import cnn_oracle as co
    order, nloc = 1, 8
    net = gb.CNN(order, N, seed=1)
    rng = np.random.default_rng(N)
    shapes, cin0, cout0 = co.layer_shapes(nloc)
    Ws = []
    for li, (taps, cout, cin) in enumerate(shapes):
        W = np.zeros((taps, cout, cin))
        src = rng.permutation(cin)[:cout] if cout <= cin else rng.integers(cin, size=cout)
        if li == 0:
            src = rng.permutation(min(nloc, cin))[:cout] if nloc >= cout else src
        W[int(rng.integers(taps)), np.arange(cout), src] = rng.choice([0.5, 1.0, 2.0], size=cout)
        Ws.append(W)
    net.set_params(np.concatenate([W.ravel() for W in Ws]).astype(np.float32))
    n = N ** 3 * nloc
    kappa = np.zeros(n)
    kappa[::nloc] = 1.0
    net.set_kappa(gb.DeviceArray.from_numpy(kappa))
    net.scale = 1.0
    r = rng.choice([-1.0, 1.0], size=n)
    z = gb.DeviceArray(n)
    net.forward(gb.DeviceArray.from_numpy(r), z)
    _, _, y = co.loss_grad(Ws, r, np.zeros(n), np.zeros(N ** 3), N, nloc, 1.0)
    ref = y[:, :nloc].ravel()
    assert np.max(np.abs(ref)) > 0
    assert np.array_equal(z.numpy(), ref)
    assert net.status() == 0


@pytest.mark.parametrize("N", [8, 16, 24])
def test_back_to_back_passes_equal_separated_ones(gb, N):
    order, nloc = 1, 8
    n = N ** 3 * nloc
    rng = np.random.default_rng(N)
    rs = [gb.DeviceArray.from_numpy(rng.uniform(-1, 1, n) * 10.0 ** k) for k in range(4)]
    t = gb.DeviceArray.from_numpy(rng.uniform(-1, 1, n))
    out = []
    for separated in (False, True):
        net = gb.CNN(order, N, seed=2)
        zs = [gb.DeviceArray(n) for _ in range(8)]
        for k in range(8):
            net.forward(rs[k % 4], zs[k])
            if separated:
                zs[k].numpy()
            if k % 3 == 2:
                net.train_step(rs[k % 4], t, 1e-2)
        out.append([z.numpy() for z in zs])
        assert net.status() == 0
    for a, b in zip(*out):
        assert np.array_equal(a, b)
    assert not np.array_equal(out[0][0], out[0][4])
