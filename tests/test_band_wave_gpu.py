"""The anti-diagonal int16 kernel against the oracle: band widths on both sides
of every class edge (8, 9, 16 or 32 lanes; 4 to 32 band indices per lane),
bands that lie in a corner of the window, one-row and one-column jobs, and
scores at the int16 limit.  Scores are whole numbers: no tolerance."""
import numpy as np
import pytest

from oracle import oracle as orc
from saber_gb300 import synth
from saber_gb300.gpu import JOB_DTYPE, Device
from saber_gb300.scoring import matrix

pytestmark = pytest.mark.gpu
B62 = matrix("BLOSUM62")
EDGES = (32, 36, 64, 128, 256, 512, 1024)


def _jobs(rng, qs, ss, widths, per):
    out = np.zeros(len(widths) * per, JOB_DTYPE)
    qlen = (qs.offsets[1:] - qs.offsets[:-1]).astype(np.int64)
    slen = (ss.offsets[1:] - ss.offsets[:-1]).astype(np.int64)
    for t in range(out.size):
        w = widths[t % len(widths)]
        q, s = int(rng.integers(qlen.size)), int(rng.integers(slen.size))
        m = int(qlen[q])
        n = int(rng.integers(1, slen[s] + 1))
        # anywhere in the m x n rectangle, corners included
        lo = int(rng.integers(-(m - 1) - w // 2, n - max(1, w // 2) + 1))
        j = out[t]
        j["query"], j["subject"] = q, s
        j["win_begin"] = int(ss.offsets[s]) + int(rng.integers(0, slen[s] - n + 1))
        j["win_len"], j["band_lo"], j["band_hi"] = n, lo, lo + w - 1
    return out


@pytest.fixture(scope="module")
def data():
    rng = np.random.default_rng(5)
    qlens = np.concatenate([[1, 2, 3, 31, 33], rng.integers(40, 1400, size=27)])
    slens = np.concatenate([[1, 2, 65], rng.integers(30, 1600, size=60)])

    def seqs(lens):
        off = np.zeros(lens.size + 1, np.uint64)
        off[1:] = np.cumsum(lens)
        return synth.ProteinSet(rng.integers(0, 24, size=int(off[-1])).astype(np.uint8), off)
    return seqs(qlens), seqs(slens)


@pytest.mark.parametrize("gaps,biased,graphs", [((11, 1), True, True), ((11, 1), False, False), ((0, 0), True, True),
                                                ((1000, 1000), False, True), ((3, 2), True, False)])
def test_class_edges_match_oracle(data, gaps, biased, graphs):
    qs, ss = data
    rng = np.random.default_rng(gaps[0] + 7)
    widths = [1, 2, 3, 4, 5, 7, 8, 9] + [e + d for e in EDGES for d in (-3, -1, 0, 1, 2)]
    jobs = _jobs(rng, qs, ss, widths, 30)
    bias = synth.query_bias(8, qs, levels=(-5, 0, 3)) if biased else None
    with Device(0) as dev:
        dev.set_scheme(B62, *gaps)
        dev.load_db(ss.codes, ss.offsets)
        dev.load_queries(qs.codes, qs.offsets, bias)
        dev.long_steps = 0
        dev.graphs = graphs
        got, st = dev.score_band_jobs(jobs)
    want, cells = orc.score_band_jobs(ss.codes, qs.codes, qs.offsets, bias, jobs, B62, *gaps, threads=4)
    assert np.array_equal(got, want), np.flatnonzero(got != want)[:10]
    assert st["banded_cells"] == cells


@pytest.mark.parametrize("jobs_n", [1210, 1230])
def test_wide_bands_on_blocks_and_on_warps(data, jobs_n):
    """Wide bands below and above the count at which they go to single warps (two per block of the launch)."""
    torch = pytest.importorskip("torch")
    qs, ss = data
    per_sm = 2 * 4 * torch.cuda.get_device_properties(0).multi_processor_count
    widths = [257, 400, 511, 512, 513, 700, 1023, 1024]
    jobs = _jobs(np.random.default_rng(jobs_n), qs, ss, widths, (jobs_n * per_sm // 1216) // len(widths) + 1)
    # bands that stay this wide when clipped to the query and the window
    qlen = (qs.offsets[1:] - qs.offsets[:-1]).astype(np.int64)
    long_q = int(np.argmax(qlen))
    long_s = int(np.argmax((ss.offsets[1:] - ss.offsets[:-1]).astype(np.int64)))
    for t in range(jobs.size):
        w = widths[t % len(widths)]
        jobs[t]["query"], jobs[t]["subject"] = long_q, long_s
        jobs[t]["win_begin"] = int(ss.offsets[long_s]) + t % 7
        jobs[t]["win_len"] = int(ss.offsets[long_s + 1] - ss.offsets[long_s]) - 7 - t % 11
        jobs[t]["band_lo"] = -(w // 2) + t % 50
        jobs[t]["band_hi"] = int(jobs[t]["band_lo"]) + w - 1
    with Device(0) as dev:
        dev.set_scheme(B62, 11, 1)
        dev.load_db(ss.codes, ss.offsets)
        dev.load_queries(qs.codes, qs.offsets, None)
        dev.long_steps = 0
        got, st = dev.score_band_jobs(jobs)
    want, cells = orc.score_band_jobs(ss.codes, qs.codes, qs.offsets, None, jobs, B62, 11, 1, threads=4)
    assert np.array_equal(got, want) and st["banded_cells"] == cells


@pytest.mark.parametrize("width", [9, 36, 90, 200, 400, 1000])
def test_scores_at_the_int16_limit(width):
    """Self-alignments whose scores lie on both sides of the limit at which a
    job is scored again in int32."""
    mat = np.full((24, 24), -400, np.int32)
    np.fill_diagonal(mat, 500)
    lens = np.array([60, 63, 64, 65, 70, 300, 1100])
    rng = np.random.default_rng(3)
    off = np.zeros(lens.size + 1, np.uint64)
    off[1:] = np.cumsum(lens)
    codes = rng.integers(0, 20, size=int(off[-1])).astype(np.uint8)
    jobs = np.zeros(lens.size, JOB_DTYPE)
    for t in range(lens.size):
        jobs[t] = (t, t, int(off[t]), int(lens[t]), -(width // 2), width - 1 - width // 2, 0)
    with Device(0) as dev:
        dev.set_scheme(mat, 900, 100)
        dev.load_db(codes, off)
        dev.load_queries(codes, off, None)
        dev.long_steps = 0
        got, st = dev.score_band_jobs(jobs)
    want, _ = orc.score_band_jobs(codes, codes, off, None, jobs, mat, 900, 100, threads=4)
    assert np.array_equal(got, want)
    assert list(want) == [500 * int(n) for n in lens] and st["i16_rescored"] == int(np.count_nonzero(want >= 32000))
