"""Tantan posteriors on both sides of the number of sequences per SM at which
the launch shape changes from two warps to eight: bit-identical to the oracle."""
import numpy as np
import pytest

from tests.test_tantan_shapes_gpu import _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("extra", [-1, 0])
def test_sequences_at_the_line(extra):
    torch = pytest.importorskip("torch")
    k = 140 * torch.cuda.get_device_properties(0).multi_processor_count + extra
    _check(np.random.default_rng(k).integers(0, 24, size=k), k)
