"""Single-sweep engine at the edges of its tiles: grids whose z extent is not a
multiple of the four nodes a thread holds (the absorber's rows are then read one
value at a time), one node beyond or short of a tile, slabs that end inside a
group of four nodes, faces without a slab, and both tile heights.  Without a
TF/SF source every engine evaluates the same expressions, so the fields equal
the per-step engine's exactly.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(n, pml, engine, rows=16, steps=19):
    from dtmaxwell4_b200 import Simulation, abi
    cfg = abi.make_config(*n, courant=0.5, absorber=abi.ABS_CPML if pml else abi.ABS_NONE, pml=pml or 0, cpml_kappa_max=3.0,
                          cpml_alpha_max=0.05)
    s = Simulation(cfg)
    rng = np.random.default_rng(5)
    mats = [abi.make_material(1.0), abi.make_material((4.0, 3.0, 2.5)),
            abi.make_material(1.0, poles=[(abi.POLE_DRUDE, 1.0, 0.7, 0.02, 0.0)], eps_inf=1.0)]
    idx = np.zeros(n, np.uint8)
    idx[n[0] // 3:, : n[1] // 2, n[2] // 4:] = 1
    idx[n[0] // 2 - 2:n[0] // 2 + 3, n[1] // 2 - 2:n[1] // 2 + 2, n[2] // 2 - 2:n[2] // 2 + 3] = 2
    s.set_materials(mats, idx)
    for c in range(6):
        s.set_field(c, rng.standard_normal(n).astype(np.float32))
    s.set_engine(engine)
    if engine == 3:
        s.set_tile_rows(rows)
    s.step(steps)
    out = [s.get_field(c) for c in range(6)]
    s.close()
    return out


@pytest.mark.parametrize("n,pml", [
    ((17, 33, 64), ((4, 4), (5, 3), (12, 12))),       # whole groups of four in the z slabs
    ((20, 31, 66), ((3, 4), (6, 5), (7, 9))),         # nz = 2 mod 4, slabs ending inside a group
    ((9, 16, 33), None),                              # one z node in the last tile, no absorber
    ((24, 17, 31), ((5, 0), (0, 6), (5, 5))),         # faces without a slab, nz odd
    ((12, 48, 96), ((4, 4), (16, 16), (32, 32))),     # slabs of whole tiles
    ((11, 9, 21), ((2, 2), (2, 3), (8, 9))),          # less than a tile; four cells between the z slabs
])
@pytest.mark.parametrize("rows", [16, 8])
def test_tile_edges_equal_the_per_step_engine(n, pml, rows):
    want = _run(n, pml, 1)
    got = _run(n, pml, 3, rows)
    for c in range(6):
        assert np.array_equal(got[c], want[c]), (c, np.abs(got[c] - want[c]).max())
