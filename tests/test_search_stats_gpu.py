"""The search's stage times: the parts add up to the total, every stage that ran
has a time, and what lies inside a part is no longer than it (device and host
clocks differ by less than 5 % + 0.2 ms)."""
import pytest

from saber_gb300 import synth
from saber_gb300 import triage as tr
from saber_gb300.gpu import Device
from saber_gb300.search import Searcher, SearchParams

pytestmark = pytest.mark.gpu
PARTS = ("t_prep_ms", "t_scan_ms", "t_triage_ms", "t_plan_ms", "t_score_ms", "t_finish_ms")


def _inside(inner, outer):
    return 0 < inner <= 1.05 * outer + 0.2


@pytest.mark.parametrize("mode", ["plain", "collecting", "triaged", "exhaustive"])
def test_stage_times(mode):
    qs, ss, _ = synth.protein_db(3, 40, 3000, planted_frac=0.2)
    with Device(0) as dev:
        kw = {"exhaustive": True} if mode == "exhaustive" else {}
        se = Searcher(dev, ss.codes, ss.offsets, SearchParams("default", masking="none", **kw))
        se.search(qs.codes, qs.offsets)
        if mode == "triaged":
            dev.set_triage(tr.init_model(1), -1e30)
        if mode == "collecting":
            tr.collect(se, qs.codes, qs.offsets)
        else:
            se.search(qs.codes, qs.offsets)
        c = se.counters
    assert abs(sum(c[k] for k in PARTS) - c["t_total_ms"]) < 1e-6 * c["t_total_ms"] + 1e-6
    assert all(c[k] >= 0 for k in PARTS)
    assert (c["t_triage_ms"] > 0) == (mode in ("collecting", "triaged"))
    for k in ("t_score_build_ms", "t_score_calls_ms", "t_score_device_ms"):
        assert _inside(c[k], c["t_score_ms"]), (k, c[k], c["t_score_ms"])
    assert _inside(c["t_finish_order_ms"], c["t_finish_ms"]) and _inside(c["t_finish_tb_ms"], c["t_finish_ms"])
    if mode != "exhaustive":
        assert c["t_plan_ms"] > 0 and c["band_rescored"] > 0
        assert _inside(c["t_score_stage2_ms"], c["t_score_ms"])
