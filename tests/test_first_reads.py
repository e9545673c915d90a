"""The first large reads of a program, before the threaded read has its pinned slots."""
import gc
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_reads_before_and_after_the_slots_are_made():
    """8.4 MB reads across the 64 MB from which the slots serve them."""
    from dtmaxwell4_b200 import Simulation, abi
    s = Simulation(abi.make_config(128, 128, 128, absorber=abi.ABS_NONE, pml=0))
    a = [np.random.default_rng(c).standard_normal(s.shape).astype(np.float32) for c in range(6)]
    for c in range(6):
        s.set_field(c, a[c])
    for q in range(10):
        assert np.array_equal(s.get_field(q % 6), a[q % 6]), q
    s.close()


def test_cost_of_a_first_read():
    """The first 8.4 MB read of a program into new pages takes at most 2.5 of a later one
    that takes the same path (pinning the slots takes 3 ms and more: 4.5 of the reads
    through them)."""
    from dtmaxwell4_b200 import Simulation, abi
    gc.collect()
    best = 1e9
    for _ in range(6):
        s = Simulation(abi.make_config(128, 128, 128, absorber=abi.ABS_NONE, pml=0))
        s.sync()
        keep, t = [], []
        for _ in range(3):
            a = time.perf_counter()
            keep.append(s.get_field(2))
            t.append(time.perf_counter() - a)
        best = min(best, t[0] / min(t[1:]))
        s.close()
    assert best <= 2.5, best
