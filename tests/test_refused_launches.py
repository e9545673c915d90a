"""A kernel that could not be launched is reported by the call that needed it.

dtmx_fail_next refuses one launch after another on the host: every call that
launches kernels returns DTMX_ERR_CUDA for each of its launches, never the
contents of a buffer that nothing has written.  Reads leave the state as it is, so the
same read afterwards gives the right values, and so does a run of 16 steps whose
graph could not be made.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = (20, 18, 21)                     # rows of 21 are padded on the device


def _sim(engine=0):
    from dtmaxwell4_b200 import Simulation, abi
    s = Simulation(abi.make_config(*N, courant=0.5, pml=4, probe_capacity=64))
    rng = np.random.default_rng(1)
    s.set_design((7, 6, 8), rng.uniform(1.0, 4.0, size=(3, 4, 5, 4)).astype(np.float32))
    s.add_point_source(abi.PointSource(comp=abi.EZ, i=6, j=9, k=10, waveform=abi.WAVE_GAUSS_SINE, amp=1.0, f0=0.05, tau=15.0, t0=10.0))
    s.add_probe(abi.EZ, 12, 9, 10)
    s.flux = s.add_flux_box((5, 5, 5), (13, 12, 14), [0.3, 0.4])
    s.dft = s.add_dft_plane(0, 8, (1 << abi.EY) | (1 << abi.HZ), [0.3, 0.5])
    for c in range(6):
        s.set_field(c, rng.standard_normal(N).astype(np.float32))
    s.set_engine(engine)
    return s


def _refused(s, call, k):
    from dtmaxwell4_b200 import abi
    from dtmaxwell4_b200.engine import DtmxError
    s.fail_next(abi.FAIL_LAUNCH, k)
    with pytest.raises(DtmxError) as e:
        call(s)
    assert e.value.code == abi.ERR_CUDA
    assert "launch" in str(e.value) or "far field" in str(e.value)


def _launches(s, call):
    n = s.launches()
    call(s)
    return s.launches() - n


READS = {
    "get_field": lambda s: s.get_field(2),
    "read_dft": lambda s: s.read_dft(s.dft),
    "read_flux": lambda s: s.read_flux(s.flux)[0],
    "far_field": lambda s: s.far_field(s.flux, [0.5, 1.0], [0.1, 2.0])[0],
    "check_finite": lambda s: np.array(s.check_finite()),
}


@pytest.mark.parametrize("name", sorted(READS))
def test_reads(name):
    read = READS[name]
    a = _sim()
    a.step(5)
    n = _launches(a, read)
    assert n >= 1
    a.close()
    a = _sim()
    a.step(5)                        # (the spectra's samples are not folded yet)
    want = read(a)
    a.close()
    for k in range(n):
        s = _sim()
        s.step(5)
        _refused(s, read, k)
        assert np.array_equal(read(s), want), k
        s.close()


def test_set_field():
    s = _sim()
    f = np.ones(N, np.float32)
    n = _launches(s, lambda q: q.set_field(1, f))
    for k in range(n):
        _refused(s, lambda q: q.set_field(1, f), k)
    s.set_field(1, f)
    assert np.array_equal(s.get_field(1), f)
    s.close()


@pytest.mark.parametrize("engine", [0, 1, 3])
def test_steps(engine):
    a = _sim(engine)
    n = _launches(a, lambda s: s.step(1))
    a.close()
    for k in range(n):
        s = _sim(engine)
        _refused(s, lambda q: q.step(1), k)
        s.close()


@pytest.mark.parametrize("engine", [0, 1, 3])
def test_a_graph_that_was_not_made_changes_nothing(engine):
    a = _sim(engine)
    n = _launches(a, lambda s: s.step(16))
    want = [a.get_field(c) for c in range(6)]
    spectrum = a.read_dft(a.dft)
    a.close()
    for k in range(n):
        s = _sim(engine)
        _refused(s, lambda q: q.step(16), k)
        s.step(16)
        for c in range(6):
            assert np.array_equal(s.get_field(c), want[c]), (k, c)
        assert np.array_equal(s.read_dft(s.dft), spectrum), k
        s.close()


@pytest.mark.parametrize("engine,order,history", [(0, 2, True), (1, 2, False), (1, 4, True)])
def test_gradients(engine, order, history):
    """One launch of a gradient run in seven is refused in turn (order 4: the two-pass adjoint)."""
    from dtmaxwell4_b200 import Simulation, abi

    def make():
        s = Simulation(abi.make_config(*N, courant=0.4, order=order, pml=4))
        s.set_design((7, 6, 8), np.full((3, 4, 5, 4), 2.0, np.float32))
        s.set_field(2, np.random.default_rng(2).standard_normal(N).astype(np.float32))
        s.set_engine(engine)
        s.set_adjoint_memory(-1 if history else 0)
        return s
    run = lambda q: q.forward_adjoint(4, 15, 0.4, 2)
    a = make()
    n = _launches(a, run)
    a.close()
    for k in range(0, n, 7):
        s = make()
        _refused(s, run, k)
        s.close()
