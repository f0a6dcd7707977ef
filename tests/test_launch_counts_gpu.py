"""library_launches of a scoring call: one kernel where one block sorts the
keys, else histogram, sum and a pass per digit of the key bits that matter (the
counts of a launch list of these calls)."""
import pytest

from saber_gb300 import synth
from saber_gb300.gpu import Device
from saber_gb300.scoring import matrix

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graphs", [True, False])
def test_sort_kernels_are_counted(graphs):
    qs, ss, planted = synth.protein_db(1, 40, 3000)
    with Device(0) as dev:
        dev.set_scheme(matrix("BLOSUM62"), 11, 1)
        dev.load_db(ss.codes, ss.offsets)
        dev.load_queries(qs.codes, qs.offsets, None)
        dev.graphs = graphs
        # (jobs, threshold): without strips 28 key bits, with them 64
        for n, steps, want in ((500, None, 1), (500, 4096, 1), (3001, None, 6), (3001, 4096, 10), (20000, None, 6)):
            if steps is not None:
                dev.long_steps = steps
            else:
                dev.long_steps = 0xFFFFFFFE
            _, st = dev.score_band_jobs(synth.band_jobs(3, qs, ss, planted, n, half_min=4, half_max=64))
            assert st["library_launches"] == want, (n, steps)
