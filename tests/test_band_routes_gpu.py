"""Which kernel a batch's bands go to in the automatic mode: batches of bands
that are wide for their queries' lengths, or wider than the anti-diagonal
kernel takes, stay on the strip kernel's lanes once there are enough of them;
ordinary bands and small batches do not.  Scores against the oracle are whole
numbers: no tolerance."""
import numpy as np
import pytest

from oracle import oracle as orc
from saber_gb300.gpu import JOB_DTYPE, Device
from saber_gb300.scoring import matrix

pytestmark = pytest.mark.gpu
B62 = matrix("BLOSUM62")


def _jobs(rng, n, qlen, slen, half, nq, ns):
    j = np.zeros(n, JOB_DTYPE)
    j["query"], j["subject"] = rng.integers(0, nq, n), rng.integers(0, ns, n)
    j["win_begin"], j["win_len"] = j["subject"].astype(np.uint64) * slen, slen
    mid = (slen - qlen) // 2 + rng.integers(-9, 10, n)
    j["band_lo"], j["band_hi"] = mid - half, mid + half
    return j


def _check(qlen, slen, batches, long_steps=None):
    rng = np.random.default_rng(qlen + slen)
    nq, ns = 17, 60
    q = rng.integers(0, 24, nq * qlen).astype(np.uint8)
    s = rng.integers(0, 24, ns * slen).astype(np.uint8)
    qo, so = (np.arange(k + 1, dtype=np.uint64) * n for k, n in ((nq, qlen), (ns, slen)))
    out = []
    with Device(0) as dev:
        dev.set_scheme(B62, 11, 1)
        dev.load_db(s, so)
        dev.load_queries(q, qo, None)
        if long_steps is not None:
            dev.long_steps = long_steps
        for n, half in batches:
            jobs = _jobs(rng, n, qlen, slen, half, nq, ns)
            want, cells = orc.score_band_jobs(s, q, qo, None, jobs, B62, 11, 1, threads=8)
            for graphs in (True, False):
                dev.graphs = graphs
                got, st = dev.score_band_jobs(jobs)
                assert np.array_equal(got, want), (n, half, graphs, np.flatnonzero(got != want)[:10])
                assert st["banded_cells"] == cells
                out.append((st["fast_jobs"], st["generic_jobs"], st["kernel_launches"], graphs))
    return out


def test_bands_above_the_anti_diagonal_kernels_width():
    # 30 rows x 1,201: 200 jobs are the int32 kernel's, 12,000 the strips'
    small, big = _check(30, 2000, [(200, 600), (12000, 600)])[::2]
    assert small[:2] == (0, 200) and big[:2] == (12000, 0)


def test_bands_wide_for_their_queries():
    # 30 rows x 401: the strip launches are part of the graph of the larger batch only
    small, _, big, _ = _check(30, 500, [(2000, 200), (20000, 200)])
    assert small == (2000, 0, 4, True) and big == (20000, 0, 6, True)


def test_ordinary_bands_stay_on_the_anti_diagonal_kernel():
    for r in _check(250, 400, [(3000, 64), (20000, 64)])[::2]:
        assert r[2] == 4


def test_a_set_threshold_holds_for_every_width():
    for r in _check(30, 2000, [(12000, 600)], long_steps=0):
        assert r[:2] == (0, 12000)
