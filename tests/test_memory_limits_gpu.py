"""Calls while most of the GPU's memory is taken: what does not fit is refused
with an error, and the handle goes on working."""
import contextlib

import numpy as np
import pytest

from oracle import oracle as orc
from saber_gb300 import presets, synth
from saber_gb300.gpu import Device, SaberGpuError, scan_params
from saber_gb300.masking import TantanParams
from saber_gb300.scoring import matrix
from tests.test_scan_gpu import _check
from tests.test_scan_small_batch_gpu import _sets

pytestmark = pytest.mark.gpu
B62 = matrix("BLOSUM62")
GIB = 1 << 30


@contextlib.contextmanager
def memory_left(leave):
    """Holds the GPU's free memory but `leave` bytes."""
    torch = pytest.importorskip("torch")
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    held = torch.empty(max(free - leave, 0), dtype=torch.uint8, device="cuda")
    try:
        yield
    finally:
        del held
        torch.cuda.empty_cache()


def test_a_refused_allocation_does_not_fail_the_next_call():
    qs, ss, planted = synth.protein_db(5, 6, 300)
    jobs = synth.band_jobs(6, qs, ss, planted, 200)
    big = np.zeros(3 * GIB, np.uint8)  # (never read: the allocation comes first)
    with Device(0) as dev:
        dev.set_scheme(B62, 11, 1)
        with memory_left(2 * GIB):
            with pytest.raises(SaberGpuError, match="allocation"):
                dev.load_db(big, np.array([0, big.size], np.uint64))
        dev.load_db(ss.codes, ss.offsets)
        dev.load_queries(qs.codes, qs.offsets, None)
        got, _ = dev.score_band_jobs(jobs)
    want, _ = orc.score_band_jobs(ss.codes, qs.codes, qs.offsets, None, jobs, B62, 11, 1, threads=4)
    assert np.array_equal(got, want)


def test_scan_after_parameters_whose_tables_did_not_fit():
    """The database state of the parameters before is built anew, not taken
    from what the refused call left of it."""
    qs, ss, _ = synth.protein_db(7, 12, 800)
    amap, asz = presets.alphabet_map()
    full, fsz = presets.full_alphabet()
    n = int(ss.codes.size)
    kw = dict(min_ids=27, exact_weight=2, db_length=n)
    gp, op = scan_params(amap, asz, presets.DS16, **kw), orc.make_scan_params(amap, asz, presets.DS16, **kw)
    # 20^7 codes: 5 GB of counts
    wide = scan_params(full, fsz, ["1111111"], min_ids=12, exact_weight=1, db_length=n)
    with Device(0) as dev:
        dev.set_scheme(B62, 11, 1)
        dev.load_db(ss.codes, ss.offsets)
        dev.load_queries(qs.codes, qs.offsets, None)
        dev.scan(gp, None, None)
        with memory_left(3 * GIB):
            with pytest.raises(SaberGpuError, match="allocation"):
                dev.scan(wide, None, None)
        got, gst = dev.scan(gp, None, None)
    want, ost = orc.scan_regions(ss.codes, ss.offsets, None, qs.codes, qs.offsets, None, None, None, B62, op)
    assert want.size > 0
    _check(got, gst, want, ost)


def test_scan_without_room_for_its_entries_windows():
    """A batch whose window records are copied to its seed entries (1 GB of
    copies) is scanned without the copies where they do not fit."""
    qn = (64 << 20) // 32 + 1
    qs, ss, _ = _sets(11, qn, 3000)
    amap, asz = presets.alphabet_map()
    kw = dict(min_ids=27, exact_weight=2, db_length=int(ss.codes.size))
    gp, op = scan_params(amap, asz, presets.DS16, **kw), orc.make_scan_params(amap, asz, presets.DS16, **kw)
    with Device(0) as dev:
        dev.set_scheme(B62, 11, 1)
        dev.load_db(ss.codes, ss.offsets)
        dev.load_queries(qs.codes, qs.offsets, None)
        with memory_left(3 * GIB // 2):
            got, gst = dev.scan(gp, None, None)
        again, ast = dev.scan(gp, None, None)  # with them
    want, ost = orc.scan_regions(ss.codes, ss.offsets, None, qs.codes, qs.offsets, None, None, None, B62, op)
    assert ost["hits"] > 0
    _check(got, gst, want, ost)
    _check(again, ast, want, ost)


@pytest.mark.parametrize("left", [2600 << 20, 600 << 20])
@pytest.mark.parametrize("longest", [900, 700_000])
def test_tantan_rows_in_less_memory(left, longest):
    """12 M residues want 3.2 GB of rows; with less they go in smaller launches."""
    rng = np.random.default_rng(4)
    lens = np.append(rng.integers(1, 900, size=26_700), longest)
    off = np.zeros(lens.size + 1, np.uint64)
    off[1:] = np.cumsum(lens)
    codes = rng.integers(0, 24, size=int(off[-1])).astype(np.uint8)
    for s in range(0, codes.size - 40, 997):
        codes[s:s + 30] = np.resize(codes[s:s + 3], 30)
    with Device(0) as dev:
        with memory_left(left):
            m, p, n, _ = dev.tantan_mask(TantanParams(), B62, codes, off, want_probs=True)
    with Device(0) as dev:
        wm, wp, wn, _ = dev.tantan_mask(TantanParams(), B62, codes, off, want_probs=True)
    assert n == wn > 0 and np.array_equal(m, wm) and np.array_equal(p.view(np.uint32), wp.view(np.uint32))


@pytest.mark.parametrize("held", ["tantan rows", "entry windows"])
def test_scratch_kept_for_speed_is_given_back_for_a_database(held):
    """A database that fits only without what the call before kept."""
    with Device(0) as dev:
        dev.set_scheme(B62, 11, 1)
        if held == "tantan rows":
            left, size = 3 * GIB, 5 * GIB // 2
            off = np.arange(0, 12_000_001, 400, dtype=np.uint64)
            codes = np.resize(np.arange(20, dtype=np.uint8), int(off[-1]))
        else:
            left, size = 6 * GIB, 4900 << 20
            qs, ss, _ = _sets(11, (64 << 20) // 32 + 1, 3000)
            amap, asz = presets.alphabet_map()
            gp = scan_params(amap, asz, presets.DS16, min_ids=27, exact_weight=2, db_length=int(ss.codes.size))
        with memory_left(left):
            if held == "tantan rows":
                dev.tantan_mask(TantanParams(), B62, codes, off)
            else:
                dev.load_db(ss.codes, ss.offsets)
                dev.load_queries(qs.codes, qs.offsets, None)
                dev.scan(gp, None, None)
            dev.load_db(np.zeros(size, np.uint8), np.array([0, size], np.uint64))
