"""The warm-start network's training kernels at the edges of their tiles."""
import numpy as np
import pytest

from mlp_oracle import NIN, NPARAM, gradient as orc_gradient

pytestmark = pytest.mark.gpu


# one row, a tile and its neighbours, one more tile than the update loads at once
@pytest.mark.parametrize("n", [1, 127, 129, 32 * 128 + 5])
def test_gradient_and_update(n):
    from graphics_b200.warmstart import WarmStartNet
    rng = np.random.default_rng(n)
    w = rng.normal(0, 0.25, NPARAM).astype(np.float32)
    norm = np.concatenate([rng.normal(0, 0.5, NIN), rng.uniform(0.5, 2, NIN), [0.2, 1.5]]).astype(np.float32)
    X = rng.normal(0, 1, (n, NIN)).astype(np.float32)
    y = rng.normal(0, 1, n).astype(np.float32)
    net = WarmStartNet(device=0, dataset_cap=n + 7, seed=0)
    net.set_params(w)
    net.set_norm(norm)
    gg, lg = net.gradient(X, y)
    go, lo = orc_gradient(w, norm.astype(np.float64), X, y)
    # a product of three BF16-rounded factors (2^-9 each) and a tanh to 2^-11
    scale = np.max(np.abs(go))
    assert abs(lg - lo) <= 1e-2 * lo + 1e-6
    for a, b in ((0, 1024), (1024, 1088), (1088, 5184), (5184, 5248), (5248, 5312), (5312, 5313)):
        assert np.max(np.abs(gg[a:b] - go[a:b])) <= 1e-2 * max(np.max(np.abs(go[a:b])), 1e-3 * scale), (a, b)
    # one step of Adam from rest with that gradient: lr g / (|g| + eps), to a
    # few roundings of the step (1e-6 of 1e-2) and of the weight (2^-24 of 1)
    net.set_dataset(X, y)
    loss = net.train(epochs=1, batch=n, lr=1e-2)
    g = gg.astype(np.float64)
    want = w - 1e-2 * g / (np.abs(g) + 1e-8)
    np.testing.assert_allclose(net.params(), want, rtol=0, atol=2e-7)
    assert loss[0] == np.float32(lg)
    net.close()
