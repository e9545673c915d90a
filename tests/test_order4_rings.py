"""Order-4 kernels with rings of 3 and of 4 stages: walks shorter than, as long as and
longer than the ring, launches on both sides of the line between the two, both
geometries, against the same grid in pieces of another length (every ring and cut
evaluates the same expressions, so the fields are equal bit for bit) and, on a
small grid, against the FP64 oracle.

Tolerance against the oracle: relative L2 2e-6 per field, FP32 rounding of 20 steps.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(cfg, planes, steps=5, rnd=3):
    from dtmaxwell4_b200 import Simulation
    s = Simulation(cfg)
    n = (cfg.nx, cfg.ny, cfg.nz)
    rng = np.random.default_rng(rnd)
    for c in range(6):
        s.set_field(c, rng.standard_normal(n).astype(np.float32))
    s.set_engine(1)
    s.set_xchunk(planes)
    s.step(steps)
    out = [s.get_field(c) for c in range(6)]
    s.close()
    return out


def _cfg(n, kind):
    from dtmaxwell4_b200 import abi
    if kind == "reference":
        return abi.make_config(*n, dx=0.005, dt=0.002, order=4, geometry=abi.GEOM_REFERENCE, absorber=abi.ABS_SPLIT_PML,
                               pml=((6, 6), (9, 9), (0, 7)), spml_vmax=0.6)
    return abi.make_config(*n, courant=0.4, order=4, absorber=abi.ABS_CPML if kind == "cpml" else abi.ABS_NONE, pml=5 if kind == "cpml" else 0)


@pytest.mark.parametrize("n,kind", [((33, 36, 40), "reference"), ((31, 35, 41), "cpml"), ((9, 18, 33), "none")])
def test_cuts_of_a_small_grid(n, kind):
    cfg = _cfg(n, kind)
    want = _run(cfg, 7)                          # 3 stages
    for planes in (1, 2, 3, 4, 5, 8, 9, 13, 64, 0):
        got = _run(cfg, planes)
        for c in range(6):
            assert np.array_equal(got[c], want[c]), (planes, c)


@pytest.mark.parametrize("n,kind", [((300, 200, 50), "none"), ((80, 264, 200), "cpml"), ((198, 201, 70), "reference")])
def test_large_launches(n, kind):
    """Automatic pieces of more than four waves (4 stages) against pieces of 7 planes of
    fewer CTAs (3 stages)."""
    cfg = _cfg(n, kind)
    want, got = _run(cfg, 7, 3), _run(cfg, 0, 3)
    for c in range(6):
        assert np.array_equal(got[c], want[c]), c


@pytest.mark.parametrize("planes", [3, 8, 20])
def test_against_the_oracle(planes):
    import pyoracle
    n = (22, 19, 37)
    cfg = _cfg(n, "cpml")
    o = pyoracle.OracleSim(cfg, "f64")
    rng = np.random.default_rng(3)
    for c in range(6):
        o.set_field(c, rng.standard_normal(n).astype(np.float32))
    o.step(20)
    got = _run(cfg, planes, 20)
    for grp in ((0, 1, 2), (3, 4, 5)):
        want = [o.get_field(c) for c in grp]
        ref = np.sqrt(sum(np.linalg.norm(w) ** 2 for w in want))
        for c, w in zip(grp, want):
            assert np.linalg.norm(got[c] - w) <= 2e-6 * ref, c


def test_large_grids_keep_their_copies_in_flight():
    """Without an absorber both stencils move the same bytes: an order-4 step of the
    per-step engine on 320^3 takes at most 1.25 of an order-2 one (1.35 with one
    plane in flight, 1.1 with two)."""
    import time
    from dtmaxwell4_b200 import Simulation, abi
    t = {}
    for order in (2, 4):
        s = Simulation(abi.make_config(320, 320, 320, courant=0.4, order=order, absorber=abi.ABS_NONE, pml=0))
        s.set_engine(1)
        best = 1e9
        for _ in range(5):
            s.sync()
            a = time.perf_counter()
            s.step(32)
            s.sync()
            best = min(best, time.perf_counter() - a)
        t[order] = best / 32 * 1e6
        s.close()
    assert t[4] <= 1.25 * t[2], t
