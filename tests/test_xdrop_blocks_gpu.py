"""Ungapped extensions in packed blocks against the oracle: sequences that end
at every offset of a block of eight, extensions that start at the first
residue of the database and batch, x-drops from 0 to above the packed limit,
large and zero biases, codes outside the alphabet.  Regions and counters
(steps among them) are whole numbers: no tolerance."""
import numpy as np
import pytest

from oracle import oracle as orc
from saber_gb300 import presets
from saber_gb300.gpu import scan_params
from saber_gb300.scoring import matrix
from saber_gb300.synth import ProteinSet
from tests.test_scan_gpu import _check

pytestmark = pytest.mark.gpu
B62 = matrix("BLOSUM62")


def _cat(seqs):
    off = np.zeros(len(seqs) + 1, np.uint64)
    off[1:] = np.cumsum([s.size for s in seqs])
    return ProteinSet(np.concatenate(seqs).astype(np.uint8), off)


@pytest.mark.parametrize("x_drop", [0, 1, 7, 20, 300, 8000, 8001, 100000])
@pytest.mark.parametrize("levels", [None, (-100, -20, 0, 0, 0, 110)])
def test_extensions_match_oracle(dev, x_drop, levels):
    rng = np.random.default_rng(x_drop + 1)
    base = rng.integers(0, 20, size=400).astype(np.uint8)
    qs, ss = [base[:60]], [base[:61]]  # the first query and subject start at the same letter
    for n in range(30, 62):
        qs.append(base[n - 30:2 * n - 20])
    for t in range(120):
        a, n = int(rng.integers(0, 300)), int(rng.integers(9, 100))
        s = base[a:a + n].copy()
        hit = rng.random(s.size) < 0.12
        s[hit] = rng.integers(0, 30, size=int(hit.sum()))  # codes above 23 among them
        ss.append(s)
    ss.append(base)  # the database ends with a hit
    qs, ss = _cat(qs), _cat(ss)
    bias = None if levels is None else rng.choice(np.array(levels, np.int8), size=qs.codes.size)
    amap, asz = presets.full_alphabet()
    kw = dict(min_ids=0, exact_weight=0, hsp_threshold=20, x_drop=x_drop)
    gp = scan_params(amap, asz, ["11011", "1111"], db_length=int(ss.codes.size), **kw)
    op = orc.make_scan_params(amap, asz, ["11011", "1111"], db_length=int(ss.codes.size), **kw)
    dev.set_scheme(B62, 11, 1)
    dev.load_db(ss.codes, ss.offsets)
    dev.load_db_mask(None)
    dev.load_queries(qs.codes, qs.offsets, bias)
    got, gst = dev.scan(gp, None, None)
    want, ost = orc.scan_regions(ss.codes, ss.offsets, None, qs.codes, qs.offsets, bias, None, None, B62, op)
    assert want.size > 0 and ost["xdrop_steps"] > 0
    _check(got, gst, want, ost)
