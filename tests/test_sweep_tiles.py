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


# cuts: by kernel (0 per-step, 1 single sweep), equal cost or not and the planes of the longest piece
@pytest.mark.parametrize("n,pml,cuts", [
    ((70, 40, 40), ((6, 6), (6, 6), (6, 6)), ((False, 1), (False, 1))),       # one wave, pieces of one plane
    ((61, 170, 150), ((6, 6), (6, 6), (6, 6)), ((True, 12), (True, 15))),     # one wave, pieces of equal cost
    ((30, 300, 290), ((6, 5), (0, 7), (8, 8)), ((True, 15), (True, 27))),     # one wave of long pieces
    ((44, 300, 290), ((6, 5), (0, 7), (8, 8)), ((True, 22), (False, 6))),     # one wave / several
    ((20, 520, 530), ((6, 5), (0, 7), (8, 8)), ((False, 4), (False, 6))),     # several waves
    ((150, 17, 20), None, ((False, 1), (False, 1))),
])
def test_pieces_of_equal_cost(n, pml, cuts):
    """The tile columns cut into pieces of equal cost (automatic) against equal
    pieces of 7 planes and of as many as a CTA's tables hold (64 planes, in the
    single sweep), on both streaming engines."""
    from dtmaxwell4_b200 import Simulation, abi
    cfg = abi.make_config(*n, courant=0.5, absorber=abi.ABS_CPML if pml else abi.ABS_NONE, pml=pml or 0)
    rng = np.random.default_rng(3)
    fields = [rng.standard_normal(n).astype(np.float32) for _ in range(6)]
    got = []
    for engine, planes in ((1, 7), (1, 0), (3, 7), (3, 0), (1, 200), (3, 200)):
        s = Simulation(cfg)
        for c in range(6):
            s.set_field(c, fields[c])
        s.set_engine(engine)
        s.set_xchunk(planes)
        s.step(5)
        got.append([s.get_field(c) for c in range(6)])
        kernel = 0 if engine == 1 else 1
        equal, _, longest = s.work_pieces(kernel)
        if planes == 0:
            assert (equal, longest) == cuts[kernel]
        else:
            assert (equal, longest) == (False, min(planes, n[0], 64 if engine == 3 else 200))
        s.close()
    for out in got[1:]:
        for c in range(6):
            assert np.array_equal(out[c], got[0][c]), c


def test_design_nodes_in_a_material_of_huge_permittivity():
    """1/eps of the material rounds to 0 in FP32; the design permittivity replaces
    it all the same (a dispersive material's nodes keep theirs)."""
    from dtmaxwell4_b200 import Simulation, abi
    n = (20, 18, 36)
    cfg = abi.make_config(*n, courant=0.5, pml=4)
    rng = np.random.default_rng(7)
    fields = [rng.standard_normal(n).astype(np.float32) for _ in range(6)]
    idx = np.zeros(n, np.uint8)
    idx[6:14, 5:13, 8:30] = 1
    mats = [abi.make_material(1.0), abi.make_material(1e60)]
    eps = rng.uniform(1.0, 4.0, size=(3, 4, 4, 9)).astype(np.float32)
    got = []
    for engine in (1, 3):
        s = Simulation(cfg)
        s.set_materials(mats, idx)
        s.set_design((8, 7, 12), eps)
        for c in range(6):
            s.set_field(c, fields[c])
        s.set_engine(engine)
        s.step(6)
        got.append([s.get_field(c) for c in range(6)])
        s.close()
    for c in range(6):
        assert np.array_equal(got[0][c], got[1][c]), c
    e = got[0][2]
    assert (e[8:12, 7:11, 12:21] != fields[2][8:12, 7:11, 12:21]).all()
    assert np.array_equal(e[6:8, 5:13, 8:30], fields[2][6:8, 5:13, 8:30])
