"""The small-batch scan (hash bitmaps in shared memory) against the oracle on
both sides of the rules that choose it: batch sizes at the edges of its passes
(16, 8 and 4 shapes a pass, then the plain scan), shape counts and spans (one,
two, three and four window words, spans above 32), alphabets of up to 15
letters.  Regions and counters are whole numbers: no tolerance."""
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


def _sets(seed, qn, n_db=40000):
    """Subjects (some empty or tiny, ragged end) and qn query residues, a third of them copied from subjects."""
    rng = np.random.default_rng(seed)

    def cut(total, lo, hi):
        lens = []
        while total > 0:
            n = min(total, int(rng.integers(lo, hi)))
            lens.append(n)
            total -= n
        off = np.zeros(len(lens) + 1, np.uint64)
        off[1:] = np.cumsum(lens)
        return off
    soff = cut(n_db + 13, 0, 700)
    db = rng.integers(0, 22, size=int(soff[-1])).astype(np.uint8)
    qoff = cut(qn, 1, 500)
    q = rng.integers(0, 22, size=qn).astype(np.uint8)
    for i in range(0, qoff.size - 1, 3):
        a, b = int(qoff[i]), int(qoff[i + 1])
        at = int(rng.integers(0, db.size - (b - a)))
        keep = rng.random(b - a) < 0.7
        q[a:b] = np.where(keep, db[at:at + b - a], q[a:b])
    return ProteinSet(q, qoff), ProteinSet(db, soff), rng


def _compare(dev, seed, qn, shapes, alpha, n_db=40000, **kw):
    qs, ss, rng = _sets(seed, qn, n_db)
    amap, asz = alpha
    db_mask = (rng.random(ss.codes.size) < 0.03).astype(np.uint8)
    q_mask = (rng.random(qn) < 0.05).astype(np.uint8)
    gp = scan_params(amap, asz, shapes, db_length=int(ss.codes.size), **kw)
    op = orc.make_scan_params(amap, asz, shapes, db_length=int(ss.codes.size), **kw)
    dev.set_scheme(B62, 11, 1)
    dev.load_db(ss.codes, ss.offsets)
    dev.load_db_mask(db_mask)
    dev.load_queries(qs.codes, qs.offsets, None)
    got, gst = dev.scan(gp, q_mask, None)
    want, ost = orc.scan_regions(ss.codes, ss.offsets, db_mask, qs.codes, qs.offsets, None, q_mask, None, B62, op)
    assert ost["hits"] > 0
    _check(got, gst, want, ost)


@pytest.mark.parametrize("qn", [40, 1000, 16384, 16385, 32768, 32769, 65536, 65537])
def test_batch_sizes_at_the_pass_edges(dev, qn):
    _compare(dev, qn, qn, presets.DS16, presets.alphabet_map(), min_ids=27, exact_weight=2)


@pytest.mark.parametrize("shapes", [["1111"], ["110011", "10101000000011"], ["1111000000000000000011", "110000011", "11011"],
                                    ["10100000000000000000000000000111", "1111", "110101", "1100011", "100000000000000111"],
                                    ["110000000000000000000000000000011", "1111"]])
def test_shape_counts_and_spans(dev, shapes):
    _compare(dev, len(shapes), 3000, shapes, presets.alphabet_map(), min_ids=20, exact_weight=1)


@pytest.mark.parametrize("letters", [2, 14, 15, 16])
def test_alphabet_sizes(dev, letters):
    amap = [c % letters if c < 20 else 255 for c in range(24)]
    shapes = ["111011011", "1111110111"] if letters == 2 else ["11011", "1000111"]
    _compare(dev, letters, 700, shapes, (amap, letters), min_ids=22, exact_weight=1)


@pytest.mark.parametrize("qn", [(64 << 20) // 32, (64 << 20) // 32 + 1])
def test_batches_at_the_entry_window_edge(dev, qn):
    """The plain scan with window records read by position (up to 64 MB of them) and copied to the entries (above)."""
    _compare(dev, 11, qn, presets.DS16[:6], presets.alphabet_map(), n_db=3000, min_ids=27, exact_weight=2)
