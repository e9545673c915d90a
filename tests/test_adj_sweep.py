"""The single-sweep adjoint at the edges of its tiles against the FP64 oracle's
adjoint: z extents that are no multiple of four, slabs that end inside a group of
four nodes or one node beyond a tile, faces without a slab, a design region that
meets a slab, the objective's plane inside the design region, dispersive blocks.

Tolerance: relative L2 of the gradient 2e-6, FP32 rounding of 40 steps (the sweep and
the two-pass kernels measure 2.5e-7 to 9.8e-7 alike on these cases).  The number of
launches tells which of the two ran: 2 to 3 a step for the sweep, 6 to 8 for
the two-pass kernels.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _case(n, pml, lo, d, drude):
    from dtmaxwell4_b200 import abi
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

    def make(kind):
        s = kind(cfg)
        s.set_materials(mats, idx, idx, idx)
        s.set_design(lo, eps)
        for c in range(6):
            s.set_field(c, fields[c])
        return s
    return make


def _agree(got, want):
    assert abs(got[0] - want[0]) <= 1e-5 * abs(want[0])
    err = np.linalg.norm(got[1] - want[1]) / np.linalg.norm(want[1])
    print("gradient rel %.2e" % err)
    assert err <= 2e-6


# equal: pieces of equal cost in the forward sweep and in the adjoint's
@pytest.mark.parametrize("n,pml,lo,d,plane,drude,equal", [
    ((30, 33, 34), ((5, 5), (5, 5), (5, 5)), (9, 9, 9), (6, 9, 7), 22, False, (False, False)),
    ((28, 20, 31), ((4, 5), (3, 6), (7, 6)), (8, 3, 5), (9, 12, 18), 20, False, (False, False)),      # nz odd, the region inside the slabs
    ((26, 34, 66), ((4, 4), (0, 5), (12, 16)), (8, 10, 14), (8, 10, 12), 12, False, (False, False)),  # the plane cuts the region
    ((24, 17, 40), None, (6, 3, 4), (8, 9, 20), 18, False, (False, False)),
    ((40, 36, 44), ((5, 5), (5, 5), (6, 5)), (12, 12, 12), (8, 9, 11), 33, True, (False, False)),
    ((48, 150, 140), ((5, 5), (5, 5), (5, 5)), (20, 60, 60), (6, 9, 7), 40, False, (True, True)),
    ((30, 300, 290), ((5, 5), (5, 5), (5, 5)), (9, 90, 90), (6, 9, 7), 22, False, (False, True)),
])
def test_gradient_against_the_oracle(n, pml, lo, d, plane, drude, equal):
    import pyoracle
    from dtmaxwell4_b200 import Simulation
    make = _case(n, pml, lo, d, drude)
    g, o = make(Simulation), make(lambda c: pyoracle.OracleSim(c, "f64"))
    got = g.forward_adjoint(40, plane, 0.4)
    assert g.launches() <= 40 * 6.5 + 10                       # (2 or 3 of them a forward step)
    assert tuple(g.work_pieces(k)[0] for k in (1, 2)) == equal
    _agree(got, o.forward_adjoint(40, plane, 0.4))
    g.close()


@pytest.mark.parametrize("drude", [False, True])
def test_without_memory_for_the_second_psi(drude):
    """Allocations of a gradient run refused one after the other: where only the
    sweep's extra arrays do not fit, the two-pass kernels serve, with the same gradient."""
    import pyoracle
    from dtmaxwell4_b200 import Simulation, abi
    from dtmaxwell4_b200.engine import DtmxError
    args = ((40, 36, 44), ((5, 5), (5, 5), (6, 5)), (12, 12, 12), (8, 9, 11))
    make = _case(*args, drude)
    want = make(lambda c: pyoracle.OracleSim(c, "f64")).forward_adjoint(40, 33, 0.4)
    ran = {True: 0, False: 0}
    for k in range(60):
        g = make(Simulation)
        g.set_engine(1)
        first = g.launches()
        g.fail_next(abi.FAIL_ALLOC, k)
        try:
            got = g.forward_adjoint(40, 33, 0.4)
        except DtmxError as e:
            assert e.code == abi.ERR_OOM
        else:
            sweep = g.launches() - first <= 40 * 7.5
            ran[sweep] += 1
            if ran[sweep] <= 2 or not sweep:
                _agree(got, want)
        g.close()
    assert ran[False] == (15 if drude else 12) and ran[True] > 0, ran
