"""The triage network's tcgen05 inference against the float64 oracle, at the
edges of its tiles of 128 rows, of its grid of one block per SM and of a host
call's chunks, and split into smaller calls.

Tolerance: activations enter as bf16 pairs (2^-16 of each value), accumulation
is fp32 over 256 terms: 2e-5 of the largest logit leaves a factor of five over
the 4e-6 that such operands show."""
import numpy as np
import pytest

from oracle import triage as otr
from saber_gb300 import triage as tr
from saber_gb300.gpu import Device


def _rows(rng, n):
    x = np.zeros((n, 32), np.float32)
    x[:, :24] = rng.normal(0.0, 1.0, size=(n, 24)) * rng.uniform(0.2, 5.0, size=24) + rng.normal(0, 3, size=24)
    return x


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 127, 128, 129, 1000, 16511, 16513, 152 * 128, 152 * 128 + 1, 40001, 131072, 131073, 262145])
def test_logits_match_oracle(n):
    rng = np.random.default_rng(n)
    x = _rows(rng, n)
    x[:, 24:] = 7.0  # unused columns do not count
    m = tr.init_model(n, x)
    m[otr.OFF_B1:otr.OFF_W2] = rng.normal(0, 0.3, 256)
    m[otr.OFF_B2:otr.OFF_W3] = rng.normal(0, 0.3, 256)
    m[otr.OFF_B3] = 0.7
    with Device(0) as dev:
        z = dev.triage_predict(m, x)
        again = dev.triage_predict(m, x)
        small = np.concatenate([dev.triage_predict(m, x[i:i + 9000]) for i in range(0, n, 9000)])
    zo, _ = otr.forward(m, x)
    scale = np.max(np.abs(zo))
    assert np.max(np.abs(z - zo)) <= 2e-5 * scale, np.max(np.abs(z - zo)) / scale
    assert np.array_equal(z, again)
    assert np.max(np.abs(small - z)) <= 4e-5 * scale
