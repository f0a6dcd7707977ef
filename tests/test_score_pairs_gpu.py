"""Both score tables of the anti-diagonal kernel in the automatic mode: batches
on both sides of the size rule on one handle, schemes changed between calls
(the pair table is built anew), and schemes whose scores plus gap open just fit
a byte and just do not.  Scores are whole numbers: no tolerance."""
import numpy as np
import pytest

from oracle import oracle as orc
from saber_gb300 import synth
from saber_gb300.gpu import JOB_DTYPE, Device
from saber_gb300.scoring import matrix

pytestmark = pytest.mark.gpu
B62 = matrix("BLOSUM62")


def _jobs(rng, qs, ss, n):
    out = np.zeros(n, JOB_DTYPE)
    slen = (ss.offsets[1:] - ss.offsets[:-1]).astype(np.int64)
    out["query"] = rng.integers(0, qs.offsets.size - 1, size=n)
    out["subject"] = rng.integers(0, slen.size, size=n)
    out["win_begin"] = ss.offsets[out["subject"]]
    out["win_len"] = slen[out["subject"]]
    mid, half = rng.integers(-60, 61, size=n), rng.integers(2, 120, size=n)
    out["band_lo"], out["band_hi"] = mid - half, mid + half
    return out


@pytest.mark.parametrize("graphs", [True, False])
def test_tables_and_schemes_match_oracle(graphs):
    rng = np.random.default_rng(12)

    def seqs(lens):
        off = np.zeros(lens.size + 1, np.uint64)
        off[1:] = np.cumsum(lens)
        return synth.ProteinSet(rng.integers(0, 24, size=int(off[-1])).astype(np.uint8), off)
    qs, ss = seqs(rng.integers(150, 500, size=20)), seqs(rng.integers(100, 600, size=200))
    bias = synth.query_bias(3, qs, levels=(-4, 0, 2))
    top = int(B62.max())
    with Device(0) as dev:
        dev.graphs = graphs
        dev.load_db(ss.codes, ss.offsets)
        for gaps in ((11, 1), (127 - top, 2), (128 - top, 2), (7, 2)):
            dev.set_scheme(B62, *gaps)
            dev.load_queries(qs.codes, qs.offsets, bias)
            for n in (17, 3001, 17):
                jobs = _jobs(rng, qs, ss, n)
                got, _ = dev.score_band_jobs(jobs)
                want, _ = orc.score_band_jobs(ss.codes, qs.codes, qs.offsets, bias, jobs, B62, *gaps, threads=4)
                assert np.array_equal(got, want), (gaps, n, np.flatnonzero(got != want)[:10])
