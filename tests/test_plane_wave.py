"""Plane-wave corrections in rows of 128 nodes, against the FP64 oracle: boxes
whose rows are one node short of, equal to and longer than a warp's 128, narrow
boxes whose faces share nodes, both stencils, both engines, a dielectric through
the box' surface.

Tolerance: 1e-5 of the E and of the H field's norm, the bound of the other
TF/SF tests against the oracle.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,box", [
    ((36, 34, 156), ((12, 23), (11, 22), (13, 142))),     # rows of 129 and 128
    ((36, 150, 34), ((12.2, 23.3), (12.1, 139.4), (11, 22))),
    ((40, 32, 33), ((14, 16), (14, 17), (13, 20))),        # two cells thick
])
@pytest.mark.parametrize("order,engine", [(2, 1), (2, 3), (4, 1)])
def test_against_the_oracle(n, box, order, engine):
    import pyoracle
    from dtmaxwell4_b200 import Simulation, abi
    cfg = abi.make_config(*n, courant=0.5 if order == 2 else 0.4, order=order, pml=5)
    t = abi.TFSF()
    t.kind = abi.TFSF_PLANE_X
    t.box_lo[:] = [float(b[0]) for b in box]
    t.box_hi[:] = [float(b[1]) for b in box]
    t.amp, t.f0, t.tau, t.t0, t.ntime = 1.0, 0.08, 10.0, 12.0, 1
    idx = np.zeros(n, np.uint8)
    idx[:, : n[1] // 2, n[2] // 3:] = 1
    mats = [abi.make_material(1.0), abi.make_material((2.0, 3.0, 1.5))]
    g, o = Simulation(cfg), pyoracle.OracleSim(cfg, "f64")
    for s in (g, o):
        s.set_materials(mats, idx, idx, idx)
        s.set_tfsf(t)
    g.set_engine(engine)
    g.step(70)
    o.step(70)
    for grp in ((0, 1, 2), (3, 4, 5)):
        want = [o.get_field(c) for c in grp]
        ref = np.sqrt(sum(np.linalg.norm(w) ** 2 for w in want))
        assert ref > 0
        for c, w in zip(grp, want):
            assert np.linalg.norm(g.get_field(c) - w) <= 1e-5 * ref, c
    g.close()
