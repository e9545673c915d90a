"""Engine 0 (automatic): the single sweep wherever it applies, with the state
where the caller may look for it.  Every engine evaluates the same expressions
without a TF/SF source, so the fields equal the per-step engine's exactly."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = (21, 34, 45)


def _sim(engine, parkable=False, absorber=True):
    from dtmaxwell4_b200 import Simulation, abi
    s = Simulation(abi.make_config(*N, courant=0.5, absorber=abi.ABS_CPML if absorber else abi.ABS_NONE, pml=5 if absorber else 0,
                                   parkable=parkable))
    rng = np.random.default_rng(2)
    for c in range(6):
        s.set_field(c, rng.standard_normal(N).astype(np.float32))
    s.set_engine(engine)
    return s


def _fields(s):
    s.sync()
    return [s.get_field(c) for c in range(6)]


def _equal(a, b):
    for c in range(6):
        assert np.array_equal(a[c], b[c]), c


@pytest.mark.parametrize("parkable", [False, True])
@pytest.mark.parametrize("steps", [(3, 16, 18), (1,), (33, 2)])
def test_automatic_equals_the_per_step_engine(steps, parkable):
    a, b = _sim(1), _sim(0, parkable)
    for n in steps:
        a.step(n)
        b.step(n)
        _equal(_fields(b), _fields(a))
    assert b.engine_config()[0] == 0
    a.close()
    b.close()


def test_a_device_address_stays_the_state():
    """After an odd number of single-sweep steps an address is handed out: from
    then on every step leaves the state there (17 steps: a graph replay and one)."""
    a, b = _sim(1), _sim(0)
    b.step(19)
    ptr = [b.device_ptr(c)[0] for c in range(6)]
    a.step(19)
    for n in (1, 17, 16):
        a.step(n)
        b.step(n)
        assert [b.device_ptr(c)[0] for c in range(6)] == ptr
        _equal(_fields(b), _fields(a))
    b.set_engine(3)                   # the choice is the caller's again
    a.step(4)
    b.step(4)
    _equal(_fields(b), _fields(a))
    a.close()
    b.close()


def test_profiling_times_both_kernels():
    s = _sim(0)
    s.step(5)
    s.set_profiling(True)
    s.step(4)
    h, e, n = s.read_profile()
    assert n == 4 and h > 0 and e > 0
    s.set_profiling(False)
    a = _sim(1)
    a.step(9 + 20)
    s.step(20)
    _equal(_fields(s), _fields(a))
    a.close()
    s.close()


def test_steps_captured_by_the_caller():
    """Steps in a graph of the caller's, replayed an odd and an even number of
    times, against plain steps."""
    import torch
    from dtmaxwell4_b200 import Simulation, abi
    n = (61, 170, 150)
    cfg = abi.make_config(*n, courant=0.5, absorber=abi.ABS_CPML, pml=6)
    rng = np.random.default_rng(3)
    fields = [rng.standard_normal(n).astype(np.float32) for _ in range(6)]
    got = []
    for replays in (0, 3):
        s = Simulation(cfg)
        for c in range(6):
            s.set_field(c, fields[c])
        s.step(2)
        if replays:
            s.sync()
            st = torch.cuda.ExternalStream(s.stream_handle())
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g, stream=st):
                s.step(1)
            with torch.cuda.stream(st):
                for _ in range(replays):
                    g.replay()
            torch.cuda.synchronize()
        else:
            s.step(3)
        got.append([s.get_field(c) for c in range(6)])
        if replays:
            del g
        s.close()
    for c in range(6):
        assert np.array_equal(got[0][c], got[1][c]), c


@pytest.mark.parametrize("before", [2, 17])
@pytest.mark.parametrize("inside", [1, 18])
def test_captured_steps_between_plain_ones(before, inside):
    """Replays of the caller's graph and plain steps in turn: the captured steps
    find the state where the plain ones left it, after a gradient run too."""
    import torch
    from dtmaxwell4_b200 import Simulation, abi
    cfg = abi.make_config(*N, courant=0.5, absorber=abi.ABS_CPML, pml=5)
    rng = np.random.default_rng(4)
    fields = [rng.standard_normal(N).astype(np.float32) for _ in range(6)]
    eps = np.full((3, 3, 4, 5), 2.0, np.float32)
    got = []
    for graph in (False, True):
        s = Simulation(cfg)
        s.set_design((8, 14, 20), eps)
        for c in range(6):
            s.set_field(c, fields[c])
        if not graph:
            s.set_engine(1)
        s.step(before)
        s.sync()
        out = []
        if graph:
            st = torch.cuda.ExternalStream(s.stream_handle())
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g, stream=st):
                s.step(inside)
        for plain in (0, 1, 19):
            if graph:
                with torch.cuda.stream(st):
                    g.replay()
            else:
                s.step(inside)
            s.step(plain)
            out.append(_fields(s))
        s.forward_adjoint(5, 15, 0.4)
        if graph:
            with torch.cuda.stream(st):
                g.replay()
        else:
            s.step(inside)
        out.append(_fields(s))
        got.append(out)
        if graph:
            del g
        s.close()
    for a, b in zip(*got):
        _equal(b, a)
