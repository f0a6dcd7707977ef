"""Which score table a batch reads: the resident scheme's pair table from the
first job on, also after the scheme changes; a call that brings its own scheme
below and above its size rule.  Scores against the oracle are whole numbers: no
tolerance."""
import numpy as np
import pytest

from oracle import oracle as orc
from saber_gb300 import synth
from saber_gb300.gpu import Device
from saber_gb300.scoring import matrix
from tests.test_score_pairs_gpu import _jobs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graphs", [True, False])
def test_small_batches_and_calls_with_their_own_scheme(graphs):
    rng = np.random.default_rng(8)
    qs, ss, _ = synth.protein_db(4, 12, 300)
    bias = synth.query_bias(5, qs, levels=(-4, 0, 2))
    big = np.full((24, 24), -90, np.int32)
    np.fill_diagonal(big, 120)
    q = rng.integers(0, 24, 90).astype(np.uint8)
    with Device(0) as dev:
        dev.graphs = graphs
        dev.load_db(ss.codes, ss.offsets)
        for mat, gaps in ((matrix("BLOSUM62"), (11, 1)), (big, (100, 9)), (matrix("BLOSUM62"), (7, 2))):
            dev.set_scheme(mat, *gaps)
            dev.load_queries(qs.codes, qs.offsets, bias)
            for n in (1, 17, 1025):
                jobs = _jobs(rng, qs, ss, n)
                got, _ = dev.score_band_jobs(jobs)
                want, _ = orc.score_band_jobs(ss.codes, qs.codes, qs.offsets, bias, jobs, mat, *gaps, threads=4)
                assert np.array_equal(got, want), (gaps, n)
            for n in (3, 3500):  # 90 rows x 150: 12 steps a lane at about 2,200 windows
                wins = [rng.integers(0, 24, int(k)).astype(np.uint8) for k in rng.integers(1, 300, n)]
                off = np.zeros(n + 1, np.uint64)
                off[1:] = np.cumsum([w.size for w in wins])
                jobs = np.zeros(n, jobs.dtype)
                jobs["subject"], jobs["win_begin"], jobs["win_len"] = np.arange(n), off[:-1], np.diff(off)
                jobs["band_lo"], jobs["band_hi"] = -90, 300
                for own in (matrix("BLOSUM62"), big):
                    got = dev.score_windows(q, None, wins, own, 11, 1)
                    want, _ = orc.score_band_jobs(np.concatenate(wins), q, np.array([0, 90], np.uint64), None, jobs, own, 11,
                                                  1, threads=4)
                    assert np.array_equal(np.asarray(got), want), n
