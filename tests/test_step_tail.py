"""The end of a step in one launch (sources, probes, DFT samples, step counter)
and the one-launch DFT fold, against the FP64 oracle: sources on sampled and
probed nodes, several on one node, more sources than the launch's list holds
(32), windows of one point and around a block of 256, frequencies around a
chunk of 8, and reads in the middle of a 16-step cycle.

Tolerance: 1e-5 of the strongest trace / of the spectrum, the bound of the
other GPU-against-oracle tests for runs of this length.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = (24, 20, 37)


def _setup(sim, nsrc, nfreq):
    from dtmaxwell4_b200 import abi
    rng = np.random.default_rng(9)
    at = [(abi.EZ, 12, 10, 18), (abi.EZ, 12, 10, 18), (abi.EY, 12, 11, 19)]
    while len(at) < nsrc:
        at.append((int(rng.integers(3)),) + tuple(int(rng.integers(6, m - 6)) for m in N))
    for q, (c, i, j, k) in enumerate(at[:nsrc]):
        sim.add_point_source(abi.PointSource(comp=c, i=i, j=j, k=k, waveform=abi.WAVE_GAUSS_SINE, amp=1.0 + 0.1 * q, f0=0.05,
                                             tau=15.0, t0=10.0 + q))
    for p in ((abi.EZ, 12, 10, 18, 0), (abi.EY, 12, 11, 19, 0), (abi.HX, 9, 9, 9, 0), (abi.EZ, 13, 11, 18, 1)):
        sim.add_probe(*p)
    om = list(2 * np.pi * np.linspace(0.02, 0.08, nfreq))
    ids = [sim.add_dft_plane(0, 12, (1 << abi.EY) | (1 << abi.EZ) | (1 << abi.HZ), om)]         # 740 points
    return ids, om


@pytest.mark.parametrize("nsrc,nfreq", [(1, 1), (3, 8), (32, 9), (40, 64)])
def test_sources_probes_and_spectra(nsrc, nfreq):
    import pyoracle
    from dtmaxwell4_b200 import Simulation, abi
    cfg = abi.make_config(*N, courant=0.5, pml=5, probe_capacity=128)
    g, o = Simulation(cfg), pyoracle.OracleSim(cfg)
    gid, om = _setup(g, nsrc, nfreq)
    oid, _ = _setup(o, nsrc, nfreq)
    steps = 45                                    # two whole cycles and 13 steps of a third
    g.step(steps)
    o.step(steps)
    tg, to = g.read_probes(), o.read_probes(128)
    assert tg.shape == to.shape
    assert np.abs(tg - to).max() <= 1e-5 * np.abs(to).max()
    dg, do = g.read_dft(gid[0]), o.read_dft(oid[0])
    assert np.linalg.norm(dg - do) <= 1e-5 * np.linalg.norm(do)
    g.close()


@pytest.mark.parametrize("window", [(3, 1, 4, 1), (2, 5, 1, 51), (2, 16, 3, 16), (0, 20, 7, 13)])
def test_windows_and_reads_mid_cycle(window):
    """Windows of 1, 255, 256 and 260 points next to a plane of other size; a
    read after 5 steps folds early and changes nothing."""
    from dtmaxwell4_b200 import Simulation, abi
    lo1, n1, lo2, n2 = window
    n = (20, 22, 60)
    cfg = abi.make_config(*n, courant=0.5, pml=4)
    rng = np.random.default_rng(1)
    fields = [rng.standard_normal(n).astype(np.float32) for _ in range(6)]
    om = list(np.linspace(0.1, 0.4, 9))
    mask = (1 << abi.EX) | (1 << abi.HY)
    got = []
    for split in ((37,), (5, 32), (16, 21)):
        s = Simulation(cfg)
        w = s.add_dft_patch(0, 9, lo1, n1, lo2, n2, mask, om)
        a = s.add_dft_plane(0, 9, mask, om)
        b = s.add_dft_plane(2, 30, 1 << abi.EZ, om[:3])
        for c in range(6):
            s.set_field(c, fields[c])
        for q in split:
            s.step(q)
            out = (s.read_dft(w), s.read_dft(a), s.read_dft(b))
        got.append(out)
        assert np.array_equal(out[0], out[1][:, :, lo1:lo1 + n1, lo2:lo2 + n2])
        s.close()
    for out in got[1:]:
        for x, y in zip(out, got[0]):
            assert np.array_equal(x, y)


def test_thousands_of_sources():
    """Far more sources than the launch's list holds, in no order, several on one
    node: after one step from zero fields E holds their sums, added in the
    order given.  Tolerance: 2e-6 of the largest (FP32 sums of at most ten
    values)."""
    from dtmaxwell4_b200 import Simulation, abi
    n = (20, 40, 50)
    s = Simulation(abi.make_config(*n, courant=0.5, pml=4))
    rng = np.random.default_rng(4)
    want = [np.zeros(n, np.float32) for _ in range(3)]
    dt = s.cfg.dt
    for q in range(5000):
        c, i, j, k = int(rng.integers(3)), 10, int(rng.integers(8, 32)), int(rng.integers(8, 42))
        src = abi.PointSource(comp=c, i=i, j=j, k=k, waveform=abi.WAVE_GAUSS_SINE, amp=float(rng.uniform(-2, 2)), f0=0.05, tau=15.0,
                              t0=float(rng.uniform(2, 12)))
        s.add_point_source(src)
        u = 0.5 * dt - src.t0
        want[c][i, j, k] += np.float32(src.amp * np.sin(2 * np.pi * src.f0 * u) * np.exp(-(u / src.tau) ** 2))
    s.step(1)
    top = max(np.abs(w).max() for w in want)
    for c in range(3):
        assert np.abs(s.get_field(c) - want[c]).max() <= 2e-6 * top, c
    s.close()


def _step_us(make, n=48):
    import time
    s = make()
    best = 1e9
    s.step(n)
    s.sync()
    for _ in range(4):
        t = time.perf_counter()
        s.step(n)
        s.sync()
        best = min(best, (time.perf_counter() - t) / n)
    s.close()
    return 1e6 * best


def test_cost_of_a_sheet_of_sources():
    """A sheet of 128 x 128 sources is one short launch more: well below 0.3 ms a
    step (searching the whole list for each source took 4 ms)."""
    from dtmaxwell4_b200 import Simulation, abi

    def make(m):
        s = Simulation(abi.make_config(24, 150, 150, courant=0.5, pml=4))
        for q in range(m * m):
            s.add_point_source(abi.PointSource(comp=abi.EZ, i=12, j=10 + q // m, k=10 + q % m, waveform=abi.WAVE_GAUSS_SINE, amp=1e-3,
                                               f0=0.05, tau=20.0, t0=30.0))
        return s
    one, sheet = _step_us(lambda: make(1)), _step_us(lambda: make(128))
    assert sheet - one <= 300.0, (one, sheet)


@pytest.mark.parametrize("every", [1, 3])
@pytest.mark.parametrize("npr", [255, 256, 257, 1500])
def test_many_probes(npr, every):
    """Probes around and beyond a block of 256, next to fewer and to no DFT blocks,
    with a source on probed nodes: the traces are the fields' values."""
    from dtmaxwell4_b200 import Simulation, abi
    n = (20, 22, 31)
    rng = np.random.default_rng(npr)
    at = [(int(rng.integers(6)),) + tuple(int(rng.integers(0, m)) for m in n) for _ in range(npr)]
    at[npr - 1] = at[0] = (abi.EZ, 9, 10, 11)
    for plane in (False, True):
        s = Simulation(abi.make_config(*n, courant=0.5, pml=4, probe_every=every, probe_capacity=2))
        s.add_point_source(abi.PointSource(comp=abi.EZ, i=9, j=10, k=11, waveform=abi.WAVE_GAUSS_SINE, amp=1.0, f0=0.05, tau=15.0, t0=4.0))
        for c in range(6):
            s.set_field(c, rng.standard_normal(n).astype(np.float32))
        for p in at:
            s.add_probe(*p)
        if plane:
            s.add_dft_plane(0, 9, 1 << abi.EZ, [0.3])
        for sample in range(3):                   # (the third one has no room)
            s.step(every)
            f = [s.get_field(c) for c in range(6)]
            if sample < 2:
                want = np.array([f[c][i, j, k] for c, i, j, k in at])
                got = s.read_probes()
                assert got.shape == (npr, sample + 1) and np.array_equal(got[:, sample], want)
        assert s.read_probes().shape == (npr, 2)
        s.close()


def test_cost_of_many_probes():
    """20000 probes stay well below 40 us a step (one block took 100)."""
    from dtmaxwell4_b200 import Simulation, abi

    def make(npr):
        s = Simulation(abi.make_config(24, 150, 150, courant=0.5, pml=4, probe_capacity=4096))
        for q in range(npr):
            s.add_probe(q % 6, 4 + q % 16, 5 + q // 150, 3 + (q * 7) % 140)
        return s
    few, many = _step_us(lambda: make(8)), _step_us(lambda: make(20000))
    assert many - few <= 40.0, (few, many)
