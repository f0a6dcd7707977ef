"""A batch scanned in blocks of positions, each with seed tables of its own:
regions and every counter equal the oracle's whatever the block length, down to
one position, on the small-batch scan, the plain one and the one with window
records at the entries, with seeds that cross a block's end and with survivors
that overflow their buffer, so that the scan runs again from the first block.
Whole numbers: no tolerance."""
import numpy as np
import pytest

from oracle import oracle as orc
from saber_gb300 import presets
from saber_gb300.gpu import Device, scan_params
from saber_gb300.scoring import matrix
from tests.test_scan_gpu import _check
from tests.test_scan_small_batch_gpu import _sets

pytestmark = pytest.mark.gpu
B62 = matrix("BLOSUM62")


def _run(seed, qn, blocks, shapes, alpha, n_db, db_mask=True, **kw):
    qs, ss, rng = _sets(seed, qn, n_db)
    amap, asz = alpha
    dm = (rng.random(ss.codes.size) < 0.03).astype(np.uint8) if db_mask else None
    qm = (rng.random(qn) < 0.05).astype(np.uint8)
    gp = scan_params(amap, asz, shapes, db_length=int(ss.codes.size), **kw)
    op = orc.make_scan_params(amap, asz, shapes, db_length=int(ss.codes.size), **kw)
    want, ost = orc.scan_regions(ss.codes, ss.offsets, dm, qs.codes, qs.offsets, None, qm, None, B62, op)
    assert ost["hits"] > 0
    for block in blocks:
        with Device(0) as dev:  # (a new handle: its survivor buffer is the smallest)
            dev.set_scheme(B62, 11, 1)
            dev.load_db(ss.codes, ss.offsets)
            dev.load_db_mask(dm)
            dev.load_queries(qs.codes, qs.offsets, None)
            dev.scan_block = block
            for _ in range(2):
                got, gst = dev.scan(gp, qm, None)
                _check(got, gst, want, ost)
    return ost


@pytest.mark.parametrize("qn,blocks", [(40, (1, 7, 39, 40, 41)), (3001, (1000, 3000))])
def test_small_batches(qn, blocks):
    _run(qn, qn, blocks, presets.DS16, presets.alphabet_map(), 20000, min_ids=22, exact_weight=2)


def test_plain_scan():
    amap = [c % 16 if c < 20 else 255 for c in range(24)]
    _run(3, 2500, (7, 1000, 2499), ["11011", "1000111"], (amap, 16), 8000, min_ids=20, exact_weight=1)


def test_entry_windows():
    n = (64 << 20) // 32 + 1
    _run(11, n, (n - 1, 700001), presets.DS16[:3], presets.alphabet_map(), 2000, min_ids=27, exact_weight=2)


@pytest.mark.parametrize("letters", [2, 16])
def test_overflowing_survivors(letters):
    # every hit survives: more than the buffer's first million
    amap = [c % letters if c < 20 else 255 for c in range(24)]
    shapes = ["1111", "10111"] if letters == 2 else ["11", "101"]
    ost = _run(letters, 900 if letters == 2 else 3000, (0, 500), shapes, (amap, letters), 30000 if letters == 2 else 60000,
               db_mask=False, min_ids=0, exact_weight=0, seed_max_occ=1 << 30)
    assert ost["hits"] - ost["hits_filtered"] > 1 << 20
