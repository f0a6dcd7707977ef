"""Tantan posteriors of batches on both sides of the rules that choose the
launch shape (sequences per SM) and of the blocks of eight positions, four
sequences a warp: bit-identical to the oracle."""
import numpy as np
import pytest

from oracle import oracle as orc
from saber_gb300.gpu import Device
from saber_gb300.masking import TantanParams
from saber_gb300.scoring import matrix

pytestmark = pytest.mark.gpu
B62 = matrix("BLOSUM62")


def _check(lens, seed):
    rng = np.random.default_rng(seed)
    offs = np.zeros(lens.size + 1, np.uint64)
    offs[1:] = np.cumsum(lens)
    codes = rng.integers(0, 26, size=int(offs[-1])).astype(np.uint8)
    for s in range(0, codes.size - 30, 211):  # short repeats
        codes[s:s + 24] = np.resize(codes[s:s + 1 + s % 5], 24)
    with Device(0) as dev:
        m, p, n, _ = dev.tantan_mask(TantanParams(), B62, codes, offs, want_probs=True)
    wm, wp, wn = orc.tantan_mask(codes, offs, B62)
    assert np.array_equal(p.view(np.uint32), wp.view(np.uint32))
    assert np.array_equal(m, np.asarray(wm, bool)) and n == wn


@pytest.mark.parametrize("per_sm,extra", [(0, 1), (0, 5), (128, -1), (128, 0), (400, -1), (400, 0)])
def test_launch_shapes(per_sm, extra):
    torch = pytest.importorskip("torch")
    k = per_sm * torch.cuda.get_device_properties(0).multi_processor_count + extra
    _check(np.random.default_rng(k).integers(0, 24, size=k), k)


@pytest.mark.parametrize("lens", [[1], [7, 8, 9], [56, 57, 58, 0], [63, 64, 65, 66, 1], [511, 512, 513, 2, 1500]])
def test_sequence_lengths(lens):
    _check(np.array(lens), len(lens))
