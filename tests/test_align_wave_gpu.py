"""The anti-diagonal traceback kernel against the oracle's alignment: band
widths on both sides of its class edges (128, 256 and 512 band indices),
corner bands, one-residue jobs, gap costs down to zero, stop scores below, at
and above the optimum (below: the row kernel takes the job over) and scores
outside int16.  Scores, coordinates, runs and cells are whole numbers: no
tolerance."""
import numpy as np
import pytest

from oracle import oracle as orc
from saber_gb300.gpu import ALIGN_JOB_DTYPE, Device
from saber_gb300.scoring import matrix

pytestmark = pytest.mark.gpu
B62 = matrix("BLOSUM62")
KEYS = ("score", "q_start", "q_end", "s_start", "s_end", "ops", "cells")


def _pairs(rng, n):
    """Queries and subjects, two thirds of them related by substitutions and long gaps."""
    qs, ss = [], []
    for t in range(n):
        m = int(rng.choice([1, 2, 17, 33, 64, 130, 300, 700]))
        q = rng.integers(0, 24, size=m).astype(np.uint8)
        s = rng.integers(0, 24, size=int(rng.integers(1, 700))).astype(np.uint8)
        if t % 3 and m > 20:
            c = q.copy()
            hit = rng.random(m) < 0.25
            c[hit] = rng.integers(0, 20, size=int(hit.sum()))
            a, g = int(rng.integers(5, m - 5)), int(rng.integers(0, 30))
            c = np.concatenate([c[:a], rng.integers(0, 20, size=g).astype(np.uint8), c[min(m, a + int(rng.integers(0, 9))):]])
            s = np.concatenate([s[:int(rng.integers(0, 40))], c, s[:20]])
        qs.append(q)
        ss.append(s.astype(np.uint8))
    return qs, ss


def _load(dev, qs, ss, bias):
    def cat(seqs):
        off = np.zeros(len(seqs) + 1, np.uint64)
        off[1:] = np.cumsum([x.size for x in seqs])
        return np.concatenate(seqs), off
    (qc, qo), (sc, so) = cat(qs), cat(ss)
    dev.load_db(sc, so)
    dev.load_queries(qc, qo, bias)
    return qo, so


@pytest.mark.parametrize("gaps,biased", [((11, 1), True), ((11, 1), False), ((0, 0), False), ((6, 6), True), ((9, 0), False),
                                         ((1000, 1000), True)])
def test_band_widths_and_stop_scores(gaps, biased):
    rng = np.random.default_rng(31 + gaps[0])
    widths = [1, 2, 3, 4, 5, 31, 33, 127, 128, 129, 130, 255, 256, 257, 258, 511, 512, 513, 900]
    qs, ss = _pairs(rng, 5 * len(widths))
    bias = rng.integers(-4, 5, size=sum(x.size for x in qs)).astype(np.int8) if biased else None
    with Device(0) as dev:
        dev.set_scheme(B62, *gaps)
        qo, so = _load(dev, qs, ss, bias)
        jobs = np.zeros(3 * len(qs), ALIGN_JOB_DTYPE)
        want = []
        for t, (q, s) in enumerate(zip(qs, ss)):
            w = widths[t % len(widths)]
            centre = int(rng.integers(-q.size // 2, s.size // 2 + 1))
            lo, hi = centre - w // 2, centre - w // 2 + w - 1
            b = None if bias is None else bias[int(qo[t]):int(qo[t + 1])]
            full = orc.banded_align(q, s, b, B62, *gaps, lo, hi)
            best = 5 if full is None else full["score"]
            for v, stop in enumerate((2 ** 31 - 1, best, max(1, best // 2))):
                jobs[3 * t + v] = (t, t, int(so[t]), s.size, lo, hi, stop)
                want.append(orc.banded_align(q, s, b, B62, *gaps, lo, hi, stop_at=stop))
        got = dev.banded_align(jobs)
    # (gaps of 1000 never pay)
    assert any(x is None for x in want) and (gaps[0] >= 1000 or any(x is not None and len(x["ops"]) > 3 for x in want))
    for t, (a, b) in enumerate(zip(got, want)):
        assert (a is None) == (b is None), t
        if a is not None:
            assert all(a[k] == b[k] for k in KEYS), (t, widths[t // 3 % len(widths)], jobs[t], a, b)


def test_scores_outside_int16():
    mat = np.full((24, 24), -400, np.int32)
    np.fill_diagonal(mat, 500)
    rng = np.random.default_rng(2)
    seqs = [rng.integers(0, 20, size=n).astype(np.uint8) for n in (60, 63, 64, 65, 200, 900)]
    with Device(0) as dev:
        dev.set_scheme(mat, 900, 100)
        _, so = _load(dev, seqs, seqs, None)
        jobs = np.zeros(len(seqs), ALIGN_JOB_DTYPE)
        for t, s in enumerate(seqs):
            jobs[t] = (t, t, int(so[t]), s.size, -20, 20, 2 ** 31 - 1)
        got = dev.banded_align(jobs)
    for s, a in zip(seqs, got):
        b = orc.banded_align(s, s, None, mat, 900, 100, -20, 20)
        assert a["score"] == 500 * s.size and all(a[k] == b[k] for k in KEYS)
