"""Window plans, two-stage scoring and the report cut on the device
(saber_gpu_search) against the same stages in Python (tests/py_engine.py):
every branch of the plan (banded, unbanded, by cell cost), regions of one
pair that bridge and that do not, stage two switched off, the other E-value
model, bit-score and unlimited E-value cuts.  Hits are compared exactly."""
import numpy as np
import pytest

from saber_gb300 import synth
from saber_gb300.search import Searcher, SearchParams
from tests.py_engine import PyEngine
from tests.test_search_gpu import _compare

pytestmark = pytest.mark.gpu


def _repeated(seed):
    """Queries with long members, subjects holding several diverged copies of a
    query at distances below and above the bridging limit of 1,024."""
    rng = np.random.default_rng(seed)
    qs = [rng.integers(0, 20, size=n).astype(np.uint8) for n in (60, 150, 300, 700, 1400)]
    subs = [rng.integers(0, 20, size=int(rng.integers(30, 900))).astype(np.uint8) for _ in range(200)]
    for t in range(60):
        q = qs[t % len(qs)]
        parts = []
        for _ in range(int(rng.integers(1, 6))):
            c = q.copy()
            hit = rng.random(c.size) < rng.uniform(0.2, 0.55)
            c[hit] = rng.integers(0, 20, size=int(hit.sum()))
            a = int(rng.integers(0, c.size // 2))
            gap = int(rng.choice([3, 90, 600, 1500]))
            parts += [c[a:], rng.integers(0, 20, size=gap).astype(np.uint8)]
        subs.append(np.concatenate(parts))

    def cat(seqs):
        off = np.zeros(len(seqs) + 1, np.uint64)
        off[1:] = np.cumsum([s.size for s in seqs])
        return np.concatenate(seqs), off
    return cat(qs), cat(subs)


@pytest.mark.parametrize("preset,kw", [
    ("default", {"max_hsps": 5, "max_regions_per_subject": 30}),
    ("default", {"score_prefilter_band": 0}),
    ("default", {"score_prefilter_band": 60}),
    ("default", {"score_band": 0, "max_hsps": 3}),
    ("default", {"score_band": 0, "window_slack": 5}),
    ("default", {"score_band": 300, "score_prefilter_band": 4, "score_prefilter_frac": 1.0}),
    ("default", {"evalue_model": "database", "evalue": 1e-3}),
    ("default", {"evalue": 1e9, "max_target_seqs": 50}),
    ("default", {"min_bitscore": 40.0, "evalue": 1e-2}),
    ("sensitive", {"hsp_threshold": 25, "hsp_floor_fraction": 0.0, "max_candidates": 40}),
])
def test_plans_and_scores_match_python_engine(preset, kw):
    from saber_gb300.gpu import Device
    (qc, qo), (sc, so) = _repeated(len(kw) + 3)
    with Device(0) as dev:
        se = Searcher(dev, sc, so, SearchParams(preset, masking="none", **kw))
        got = se.search(qc, qo)
        want = PyEngine(se).search(qc, qo)
    assert sum(len(h) for h in want) > 0
    _compare(got, want)


def test_batch_without_regions():
    from saber_gb300.gpu import Device
    rng = np.random.default_rng(1)
    _, ss, _ = synth.protein_db(3, 4, 50)
    q = rng.integers(0, 20, size=12).astype(np.uint8)
    with Device(0) as dev:
        se = Searcher(dev, ss.codes, ss.offsets, SearchParams("default", masking="none"))
        assert se.search(q, np.array([0, 5, 5, 12], np.uint64)) == [[], [], []]
