"""The device's shuffle of a training pass gives the order of the sequential
Fisher-Yates loop with the seeded generator, pass after pass: with one sample a
step and a learning rate of nothing, each step's loss tells its sample."""
import numpy as np
import pytest

from persiansph_gb300.closure import ClosureNet

pytestmark = pytest.mark.gpu

M = (1 << 64) - 1


def draws(state):
    while True:
        state = (state + 0x9E3779B97F4A7C15) & M
        z = state
        z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & M
        z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & M
        yield z ^ (z >> 31)


@pytest.mark.parametrize("n,passes", [(1, 3), (2, 5), (3, 4), (257, 3), (1000, 2)])
@pytest.mark.parametrize("seed", [0, 12345, M])
def test_order_of_the_samples(gpu, n, passes, seed):
    net = ClosureNet(3)
    x = np.zeros((n, 6), np.float32)
    y = np.linspace(1.0, 2.0, n).astype(np.float32) if n > 1 else np.ones(1, np.float32)
    net.set_data(x, y)
    c = float(net.infer(x[:1])[0])
    losses = net.train(n * passes, batch=1, lr=1e-30, seed=seed)
    got = np.rint((c + np.sqrt(losses.astype(np.float64)) - 1.0) * max(n - 1, 0)).astype(int)
    rng, order = draws(seed), list(range(n))
    for q in range(passes):
        for i in range(n - 1, 0, -1):
            j = next(rng) % (i + 1)
            order[i], order[j] = order[j], order[i]
        assert got[q * n:(q + 1) * n].tolist() == order, f"pass {q}"
