"""Tracebacks of queries of a few rows on bands of every width: both sides of
the rule that leaves them to the row kernel, in one call.  Scores, coordinates,
runs and cells against the oracle are whole numbers: no tolerance."""
import numpy as np
import pytest

from oracle import oracle as orc
from saber_gb300.gpu import ALIGN_JOB_DTYPE, Device
from saber_gb300.scoring import matrix

pytestmark = pytest.mark.gpu
B62 = matrix("BLOSUM62")
KEYS = ("score", "q_start", "q_end", "s_start", "s_end", "ops", "cells")


@pytest.mark.parametrize("gaps", [(11, 1), (2, 0)])
def test_short_queries_on_wide_bands(gaps):
    rng = np.random.default_rng(17 + gaps[0])
    qs, ss, bands = [], [], []
    for m in (1, 2, 7, 8, 9, 16, 17, 31, 32, 40):
        for w in (1, 16, 17, 111, 128, 129, 144, 145, 256, 257, 272, 273, 511, 512, 513):
            q = rng.integers(0, 20, size=m).astype(np.uint8)
            s = rng.integers(0, 20, size=m + w + int(rng.integers(0, 30))).astype(np.uint8)
            at = int(rng.integers(0, w))
            s[at:at + m] = q
            s[at + m // 2:at + m // 2 + 1] = 23
            qs.append(q)
            ss.append(s)
            bands.append((0, w - 1))

    def cat(seqs):
        off = np.zeros(len(seqs) + 1, np.uint64)
        off[1:] = np.cumsum([x.size for x in seqs])
        return np.concatenate(seqs), off
    (qc, qo), (sc, so) = cat(qs), cat(ss)
    jobs = np.zeros(2 * len(qs), ALIGN_JOB_DTYPE)
    want = []
    for t, (q, s) in enumerate(zip(qs, ss)):
        full = orc.banded_align(q, s, None, B62, *gaps, *bands[t])
        for v, stop in enumerate((2 ** 31 - 1, 5 if full is None else full["score"])):
            jobs[2 * t + v] = (t, t, int(so[t]), s.size, *bands[t], stop)
            want.append(orc.banded_align(q, s, None, B62, *gaps, *bands[t], stop_at=stop))
    with Device(0) as dev:
        dev.set_scheme(B62, *gaps)
        dev.load_db(sc, so)
        dev.load_queries(qc, qo, None)
        got = dev.banded_align(jobs)
    for t, (a, b) in enumerate(zip(got, want)):
        assert (a is None) == (b is None), t
        if a is not None:
            assert all(a[k] == b[k] for k in KEYS), (qs[t // 2].size, bands[t // 2], a, b)
