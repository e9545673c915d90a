"""Per-step kernels at the edges of their tiles against the FP64 oracle: the
reference geometry with a mirror boundary one or two nodes into the last tile
(its images are staged in the same box), z extents that are no multiple of four,
both stencils, split PML and none; and the box geometry at order 4.

Tolerance: relative L2 2e-6 per field (E or H together): FP32 rounding of 30 steps.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _compare(cfg, mats, idx, steps=30):
    import pyoracle
    from dtmaxwell4_b200 import Simulation
    n = (cfg.nx, cfg.ny, cfg.nz)
    rng = np.random.default_rng(12)
    fields = [rng.standard_normal(n).astype(np.float32) for _ in range(6)]
    g, o = Simulation(cfg), pyoracle.OracleSim(cfg, "f64")
    for s in (g, o):
        s.set_materials(mats, idx, idx, idx)
    g.set_engine(1)
    for c in range(6):
        g.set_field(c, fields[c])
        o.set_field(c, g.get_field(c))            # (non-live nodes are held at zero)
    g.step(steps)
    o.step(steps)
    for grp in ((0, 1, 2), (3, 4, 5)):
        want = [o.get_field(c) for c in grp]
        got = [g.get_field(c).astype(np.float64) for c in grp]
        ref = np.sqrt(sum(np.linalg.norm(w) ** 2 for w in want))
        for w, v in zip(want, got):
            err = np.linalg.norm(v - w) / ref
            assert np.isfinite(err) and err <= 2e-6, (grp, err)
    g.close()


@pytest.mark.parametrize("order", [2, 4])
@pytest.mark.parametrize("n", [(9, 18, 33), (12, 33, 34), (15, 21, 31), (9, 30, 64), (18, 48, 66)])
def test_mirror_boundaries(n, order):
    from dtmaxwell4_b200 import abi
    cfg = abi.make_config(*n, dx=0.005, dt=0.002, order=order, geometry=abi.GEOM_REFERENCE, absorber=abi.ABS_NONE, pml=0)
    idx = np.zeros(n, np.uint8)
    idx[:, :, :5] = 1
    _compare(cfg, [abi.make_material(1.75 ** 2), abi.make_material((2.0, 3.0, 4.0))], idx)


@pytest.mark.parametrize("n,pml", [((36, 36, 40), ((6, 6), (9, 9), (0, 7))), ((33, 42, 45), ((9, 9), (6, 6), (0, 16)))])
def test_split_pml(n, pml):
    from dtmaxwell4_b200 import abi
    cfg = abi.make_config(*n, dx=0.005, dt=0.002, order=4, geometry=abi.GEOM_REFERENCE, absorber=abi.ABS_SPLIT_PML, pml=pml,
                          spml_vmax=0.6)
    idx = np.zeros(n, np.uint8)
    idx[:, :, :8] = 1
    drude = abi.make_material(1.0, poles=[(abi.POLE_DRUDE, 1.0, 45.0, 0.05, 0.0)], eps_inf=1.0)
    _compare(cfg, [abi.make_material(3.0), drude], idx)


@pytest.mark.parametrize("n,pml", [((14, 17, 33), ((4, 4), (5, 5), (6, 7))), ((20, 33, 64), ((4, 5), (0, 6), (12, 12))), ((11, 16, 30), None)])
@pytest.mark.parametrize("order", [2, 4])
def test_box(n, pml, order):
    from dtmaxwell4_b200 import abi
    cfg = abi.make_config(*n, courant=0.4, order=order, absorber=abi.ABS_CPML if pml else abi.ABS_NONE, pml=pml or 0, cpml_kappa_max=2.0)
    idx = np.zeros(n, np.uint8)
    idx[n[0] // 2:, 3:, n[2] // 3:] = 1
    _compare(cfg, [abi.make_material(1.0), abi.make_material((2.0, 3.0, 4.0))], idx)
