"""Second-stage decisions that the device leaves to the host: scores at the
threshold, thresholds without a value, and length adjustments at a whole number.
Hits against the Python engine, exactly."""
import math

import pytest

from saber_gb300.search import Searcher, SearchParams
from tests.py_engine import PyEngine
from tests.test_plan_gpu import _repeated
from tests.test_search_gpu import _compare

pytestmark = pytest.mark.gpu


def _both(karlin=None, **kw):
    from saber_gb300.gpu import Device
    (qc, qo), (sc, so) = _repeated(9)
    with Device(0) as dev:
        se = Searcher(dev, sc, so, SearchParams("default", masking="none", **kw))
        for k, v in (karlin or {}).items():
            setattr(se.karlin, k, v)
        got = se.search(qc, qo)
        counters = dict(se.counters)
        want = PyEngine(se).search(qc, qo)
    _compare(got, want)
    assert sum(len(h) for h in want) > 0
    return counters


@pytest.mark.parametrize("frac", [45.0, 60.0, 0.0])
def test_scores_at_the_threshold(frac):
    # an E-value that every score passes makes the bound 1, the threshold frac itself
    c = _both(evalue=1e15, score_prefilter_frac=frac, max_target_seqs=40)
    assert 0 < c["band_rescored"] <= c["band_scored_regions"]


@pytest.mark.parametrize("frac", [math.inf, -math.inf, math.nan])
def test_thresholds_without_a_value(frac):
    c = _both(score_prefilter_frac=frac)
    assert c["band_rescored"] == (c["band_scored_regions"] if frac < 0 else 0)


@pytest.mark.parametrize("beta", [-3.0, 0.0, 1.0, 30.0, 31.0])
def test_length_adjustments_at_a_whole_number(beta):
    # alpha 0: the adjustment is beta, rounded up, whatever the lengths
    _both({"alpha": 0.0, "alpha_d_lambda": 0.0, "beta": beta}, evalue=1e-3)
