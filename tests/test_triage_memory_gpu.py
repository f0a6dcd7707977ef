"""The triage network's work buffers: kept from call to call while they are
small, given back after a call on many rows (and on every way out of it)."""
import numpy as np
import pytest

from saber_gb300 import triage as tr
from saber_gb300.gpu import Device

pytestmark = pytest.mark.gpu
MB = 1 << 20


def _free():
    torch = pytest.importorskip("torch")
    return torch.cuda.mem_get_info()[0]


@pytest.mark.parametrize("call", ["predict", "grads"])
def test_buffers_of_a_large_call_are_given_back(call):
    rng = np.random.default_rng(2)
    n = 2_500_000 if call == "predict" else 100_000
    x = np.zeros((n, 32), np.float32)
    x[:1000, :24] = rng.normal(size=(1000, 24))
    x[1000:] = np.resize(x[:1000], x[1000:].shape)
    y = (np.arange(n) % 9 == 0).astype(np.uint8)
    m = tr.init_model(1, x[:1000])

    def run(dev, k):
        return dev.triage_predict(m, x[:k]) if call == "predict" else dev.triage_grads(m, x[:k], y[:k], 3.0)[0]
    with Device(0) as dev:
        small = run(dev, 2000)
        before = _free()
        run(dev, n)
        assert before - _free() < 32 * MB
        again = run(dev, 2000)
        assert np.array_equal(small, again)
