"""The int32 kernel on bands of every width up to the anti-diagonal kernel's:
jobs whose int16 score reaches the limit are scored again there, so identical
and diverged pairs under a scheme of large scores reach its rows in parallel and
its pipelined strips, from the anti-diagonal kernel and from the strips, in
captured graphs and step by step.  Scores are whole numbers: no tolerance."""
import numpy as np
import pytest

from oracle import oracle as orc
from saber_gb300.gpu import JOB_DTYPE, Device

pytestmark = pytest.mark.gpu
LIMIT = 32000


@pytest.mark.parametrize("gaps", [(900, 100), (40, 7), (0, 0)])
@pytest.mark.parametrize("biased", [False, True])
def test_rescored_bands_match_oracle(gaps, biased):
    rng = np.random.default_rng(gaps[0] + 5)
    mat = np.full((24, 24), -300, np.int32)
    np.fill_diagonal(mat, 500)
    qs, ss, jobs = [], [], []
    widths = [1, 2, 7, 8, 9, 15, 16, 17, 31, 33, 36, 64, 65, 128, 129, 200, 256, 257, 500, 512, 513, 900, 1023, 1024, 1025]
    for t, w in enumerate(widths * 4):
        m = int(rng.choice([66, 90, 140, 300, 700, 1300]))
        q = rng.integers(0, 20, m).astype(np.uint8)
        s = q.copy()
        if t % 2:  # substitutions and, on bands that hold them, a gap
            hit = rng.random(m) < 0.15
            s[hit] = rng.integers(0, 20, int(hit.sum()))
            if w > 30:
                a = int(rng.integers(10, m - 10))
                s = np.concatenate([s[:a], rng.integers(0, 20, min(w // 3, 40)).astype(np.uint8), s[a:]])
        lead = int(rng.integers(0, 30))
        s = np.concatenate([rng.integers(0, 20, lead).astype(np.uint8), s, rng.integers(0, 20, 25).astype(np.uint8)])
        qs.append(q)
        ss.append(s)
        lo = lead - int(rng.integers(0, max(1, w // 2)))
        jobs.append((t, t, 0, s.size, lo, lo + w - 1, 0))

    def cat(seqs):
        off = np.zeros(len(seqs) + 1, np.uint64)
        off[1:] = np.cumsum([x.size for x in seqs])
        return np.concatenate(seqs), off
    (qc, qo), (sc, so) = cat(qs), cat(ss)
    arr = np.array(jobs, JOB_DTYPE)
    arr["win_begin"] = so[:-1]
    bias = rng.integers(-100, 101, qc.size).astype(np.int8) if biased else None
    want, cells = orc.score_band_jobs(sc, qc, qo, bias, arr, mat, *gaps, threads=8)
    wide = np.array([w for w in widths * 4]) > 1024
    with Device(0) as dev:
        dev.set_scheme(mat, *gaps)
        dev.load_db(sc, so)
        dev.load_queries(qc, qo, bias)
        for graphs in (True, False):
            for steps in (0xFFFFFFFE, 0, 0xFFFFFFFF):
                dev.graphs, dev.long_steps = graphs, steps
                got, st = dev.score_band_jobs(arr)
                assert np.array_equal(got, want), (graphs, steps, np.flatnonzero(got != want)[:10])
                assert st["banded_cells"] == cells
                again = (want >= LIMIT) & ~wide
                assert st["i16_rescored"] >= int(again.sum()) > 40
