"""The single-sweep adjoint at the edges of its tiles against the FP64 oracle's
adjoint: z extents that are no multiple of four, slabs that end inside a group of
four nodes or one node beyond a tile, faces without a slab, a design region that
meets a slab, the objective's plane inside the design region, dispersive blocks.

Tolerance: relative L2 of the gradient 2e-6; FP32 rounding of 40 steps (the
two-pass kernels, run by the oracle-sized cases of test_adjoint, stay at 5e-7).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,pml,lo,d,plane,drude", [
    ((30, 33, 34), ((5, 5), (5, 5), (5, 5)), (9, 9, 9), (6, 9, 7), 22, False),
    ((28, 20, 31), ((4, 5), (3, 6), (7, 6)), (8, 3, 5), (9, 12, 18), 20, False),      # nz odd, the region inside the slabs
    ((26, 34, 66), ((4, 4), (0, 5), (12, 16)), (8, 10, 14), (8, 10, 12), 12, False),  # the plane cuts the region
    ((24, 17, 40), None, (6, 3, 4), (8, 9, 20), 18, False),
    ((40, 36, 44), ((5, 5), (5, 5), (6, 5)), (12, 12, 12), (8, 9, 11), 33, True),
    ((48, 150, 140), ((5, 5), (5, 5), (5, 5)), (20, 60, 60), (6, 9, 7), 40, False),   # pieces of equal cost, both sweeps
    ((30, 300, 290), ((5, 5), (5, 5), (5, 5)), (9, 90, 90), (6, 9, 7), 22, False),    # the adjoint's alone
])
def test_gradient_against_the_oracle(n, pml, lo, d, plane, drude):
    import pyoracle
    from dtmaxwell4_b200 import Simulation, abi
    cfg = abi.make_config(*n, courant=0.5, absorber=abi.ABS_CPML if pml else abi.ABS_NONE, pml=pml or 0, cpml_kappa_max=2.5,
                          cpml_alpha_max=0.04)
    rng = np.random.default_rng(8)
    mats = [abi.make_material(1.0), abi.make_material((3.0, 2.0, 4.0)),
            abi.make_material(1.0, poles=[(abi.POLE_DRUDE, 1.0, 0.6, 0.02, 0.0)], eps_inf=1.5)]
    idx = np.zeros(n, np.uint8)
    idx[:, : n[1] // 3, n[2] // 2:] = 1
    if drude:
        idx[lo[0] + d[0] - 1:lo[0] + d[0] + 6, 14:22, 15:24] = 2
    eps = rng.uniform(1.0, 6.0, size=(3,) + d).astype(np.float32)
    fields = [rng.standard_normal(n).astype(np.float32) for _ in range(6)]
    res = []
    for make in (Simulation, lambda c: pyoracle.OracleSim(c, "f64")):
        s = make(cfg)
        s.set_materials(mats, idx, idx, idx)
        s.set_design(lo, eps)
        for c in range(6):
            s.set_field(c, fields[c])
        res.append(s.forward_adjoint(40, plane, 0.4))
    (jg, gg), (jo, go) = res
    assert abs(jg - jo) <= 1e-5 * abs(jo)
    err = np.linalg.norm(gg - go) / np.linalg.norm(go)
    print("gradient rel %.2e" % err)
    assert err <= 2e-6
