"""Two databases one after the other on one handle: the triage features of the
second search are the second database's, also where both hold the same number
of residues (and so stand in the same buffer) in different subjects.  The rows
are compared bit for bit with those of a handle that has seen one database."""
import numpy as np
import pytest

from saber_gb300 import synth
from saber_gb300 import triage as tr
from saber_gb300.gpu import Device
from saber_gb300.search import Searcher, SearchParams

pytestmark = pytest.mark.gpu


def _rows(dev, codes, offsets, qs):
    se = Searcher(dev, codes, offsets, SearchParams("default", masking="none"))
    rows, _, _ = tr.collect(se, qs.codes, qs.offsets)
    return rows


@pytest.mark.parametrize("order", ["more subjects", "fewer subjects"])
def test_features_follow_the_loaded_database(order):
    qs, ss, _ = synth.protein_db(31, 20, 600, planted_frac=0.3)
    total = int(ss.codes.size)
    # the same number of residues: other letters, in three times as many subjects
    cuts = np.unique(np.concatenate([ss.offsets, np.linspace(0, total, 1200).astype(np.uint64)]))
    other = ss.codes.copy()
    other[::5] = 0
    first, second = (ss.codes, ss.offsets), (other, cuts)
    if order == "fewer subjects":
        first, second = second, first
    assert first[0].size == second[0].size
    with Device(0) as dev:
        before = _rows(dev, *first, qs)
        got = _rows(dev, *second, qs)
    with Device(0) as dev:
        want = _rows(dev, *second, qs)
    assert before.size and want.size
    assert got.shape == want.shape and np.array_equal(got.view(np.uint32), want.view(np.uint32))
