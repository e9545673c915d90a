"""Dipole TF/SF corrections with a thread a tap (small boxes) and a thread a node
(tens of thousands of corrected nodes), against the FP64 oracle: flat boxes along
each axis, so that jobs of very different lengths share a launch and the rows of
a face normal to z are a few nodes long, both stencils, a dielectric through the
surface.

Tolerance: 1e-5 of the E and of the H field's norm, the bound of the other TF/SF tests
against the oracle.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _source(n, size):
    from dtmaxwell4_b200 import abi
    t = abi.TFSF()
    t.kind = abi.TFSF_DIPOLE
    lo = [0.5 * (m - b) + 0.3 for m, b in zip(n, size)]
    t.box_lo[:] = lo
    t.box_hi[:] = [v + b for v, b in zip(lo, size)]
    t.c, t.w, t.kenv, t.tstop, t.ntime = 1.0, 2 * np.pi / 10, 0.3, 0.0, 1
    return t


@pytest.mark.parametrize("order", [2, 4])
@pytest.mark.parametrize("n,size", [
    ((30, 124, 118), (8, 102, 96)),          # a thread a node
    ((120, 32, 126), (98, 9, 104)),
    ((118, 122, 30), (96, 100, 7)),
    ((30, 70, 66), (8, 48, 44)),             # a thread a tap
    ((60, 66, 30), (38, 44, 7)),
])
def test_against_the_oracle(n, size, order):
    import pyoracle
    from dtmaxwell4_b200 import Simulation, abi
    cfg = abi.make_config(*n, courant=0.5 if order == 2 else 0.4, order=order, pml=5)
    idx = np.zeros(n, np.uint8)
    idx[:, :, : n[2] // 3] = 1
    g, o = Simulation(cfg), pyoracle.OracleSim(cfg)
    for s in (g, o):
        s.set_materials([abi.make_material(1.0), abi.make_material((2.0, 3.0, 1.5))], idx, idx, idx)
        s.set_tfsf(_source(n, size))
        s.step(50)
    for grp in ((0, 1, 2), (3, 4, 5)):
        want = [o.get_field(c) for c in grp]
        ref = np.sqrt(sum(np.linalg.norm(w) ** 2 for w in want))
        assert ref > 0
        for c, w in zip(grp, want):
            assert np.linalg.norm(g.get_field(c) - w) <= 1e-5 * ref, c
    g.close()


def test_cost_on_a_large_flat_box():
    """Order 4, a box of 170 x 170 x 10 cells: the corrections take well below 200 us a
    step (390 with eight threads a node and the shorter jobs' blocks computing too)."""
    import time
    from dtmaxwell4_b200 import Simulation, abi
    n, us = (200, 200, 40), []
    for src in (False, True):
        s = Simulation(abi.make_config(*n, courant=0.4, order=4, pml=6))
        if src:
            s.set_tfsf(_source(n, (170, 170, 10)))
        best = 1e9
        for _ in range(5):
            s.sync()
            t = time.perf_counter()
            s.step(32)
            s.sync()
            best = min(best, (time.perf_counter() - t) / 32)
        us.append(1e6 * best)
        s.close()
    assert us[1] - us[0] <= 200.0, us
