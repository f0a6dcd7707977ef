"""Calls while most of the GPU's memory is taken: what does not fit is refused
with an error, and the handle goes on working."""
import contextlib

import numpy as np
import pytest

from oracle import oracle as orc
from saber_gb300 import synth
from saber_gb300.gpu import Device, SaberGpuError
from saber_gb300.scoring import matrix

pytestmark = pytest.mark.gpu
B62 = matrix("BLOSUM62")
GIB = 1 << 30


@contextlib.contextmanager
def memory_left(leave):
    """Holds the GPU's free memory but `leave` bytes."""
    torch = pytest.importorskip("torch")
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    held = torch.empty(max(free - leave, 0), dtype=torch.uint8, device="cuda")
    try:
        yield
    finally:
        del held
        torch.cuda.empty_cache()


def test_a_refused_allocation_does_not_fail_the_next_call():
    qs, ss, planted = synth.protein_db(5, 6, 300)
    jobs = synth.band_jobs(6, qs, ss, planted, 200)
    big = np.zeros(3 * GIB, np.uint8)  # (never read: the allocation comes first)
    with Device(0) as dev:
        dev.set_scheme(B62, 11, 1)
        with memory_left(2 * GIB):
            with pytest.raises(SaberGpuError, match="allocation"):
                dev.load_db(big, np.array([0, big.size], np.uint64))
        dev.load_db(ss.codes, ss.offsets)
        dev.load_queries(qs.codes, qs.offsets, None)
        got, _ = dev.score_band_jobs(jobs)
    want, _ = orc.score_band_jobs(ss.codes, qs.codes, qs.offsets, None, jobs, B62, 11, 1, threads=4)
    assert np.array_equal(got, want)
