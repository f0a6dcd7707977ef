"""The triage network's gradient kernels at the edges of their 64-row tiles,
32-row blocks and row splits, against the float64 oracle.

Rows with a hidden unit within 2e-5 of its ReLU's kink are left out, so that
no rounding can switch a unit.  Tolerance: activations carry the rounding of
fp32 sums of 256 terms (about 16 x 2^-24 = 1e-6 relative), a gradient the same
again for each of its three sums; 1e-4 of a block's norm (of sum |dz| for the
output bias, whose terms cancel) leaves a factor of 30."""
import numpy as np
import pytest

from oracle import triage as otr
from saber_gb300 import triage as tr
from saber_gb300.gpu import Device

RTOL = 1e-4


def _case(n, seed):
    rng = np.random.default_rng(seed)
    k = n + 64 + n // 16
    x = np.zeros((k, 32), np.float32)
    x[:, :24] = rng.normal(0.0, 1.0, size=(k, 24)) * rng.uniform(0.2, 5.0, size=24) + rng.normal(0, 3, size=24)
    m = tr.init_model(seed, x)
    m[otr.OFF_B1:otr.OFF_W2] = rng.normal(0, 0.05, 256)
    m[otr.OFF_B2:otr.OFF_W3] = rng.normal(0, 0.05, 256)
    _, (xn, h1, _, p) = otr.forward(m, x)
    near = np.minimum(np.abs(xn @ p["W1"] + p["b1"]).min(axis=1), np.abs(h1 @ p["W2"] + p["b2"]).min(axis=1))
    x = x[near > 2e-5][:n]
    assert x.shape[0] == n
    return m, x, (rng.random(n) < 0.2).astype(np.uint8)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 31, 32, 33, 64, 65, 127, 128, 129, 257, 1000, 4096, 4129, 9001])
def test_gradients_at_tile_and_split_edges(n):
    m, x, y = _case(n, 100 + n)
    with Device(0) as dev:
        for _ in range(2):  # the second pass reuses the handle's buffers
            g, loss = dev.triage_grads(m, x, y, 5.0)
    lo, go = otr.loss_and_grads(m, x, y, 5.0)
    assert abs(loss - lo) <= 1e-5 * max(1.0, abs(lo))
    z, _ = otr.forward(m, x)
    dz = np.where(y > 0, 5.0, 1.0) * (1.0 / (1.0 + np.exp(-z)) - y) / n
    for name, a, b in (("W1", 0, otr.OFF_B1), ("b1", otr.OFF_B1, otr.OFF_W2), ("W2", otr.OFF_W2, otr.OFF_B2),
                       ("b2", otr.OFF_B2, otr.OFF_W3), ("W3", otr.OFF_W3, otr.OFF_B3)):
        assert np.linalg.norm(g[a:b] - go[a:b]) <= RTOL * np.linalg.norm(go[a:b]), (n, name)
    assert abs(g[otr.OFF_B3] - go[otr.OFF_B3]) <= RTOL * np.abs(dz).sum()
    assert not np.any(g[otr.OFF_MU:])
