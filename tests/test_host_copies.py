"""Fields and spectra between the device and host memory of every kind: rows
that are padded on the device, more than one piece of the threaded read (1 MB
pieces from 4 MB on), pinned memory, and reads of two contexts at once."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def slots():
    """The threaded read's pinned slots: made by a read of 32 MB, kept while a context
    lives."""
    from dtmaxwell4_b200 import Simulation, abi
    s = Simulation(abi.make_config(512, 128, 128, absorber=abi.ABS_NONE, pml=0))
    a = np.random.default_rng(1).standard_normal(s.shape).astype(np.float32)
    s.set_field(0, a)
    assert np.array_equal(s.get_field(0), a)      # 33.6 MB
    yield
    s.close()


@pytest.mark.parametrize("n", [(9, 8, 11), (64, 161, 103), (40, 64, 512), (1100, 33, 31)])
def test_field_roundtrip(n):
    import torch
    from dtmaxwell4_b200 import Simulation, abi
    s = Simulation(abi.make_config(*n, absorber=abi.ABS_NONE, pml=0))
    rng = np.random.default_rng(4)
    a = [rng.standard_normal(n).astype(np.float32) for _ in range(2)]
    for c in (0, 4):
        s.set_field(c, a[c // 4])
    pinned = torch.empty(n, dtype=torch.float32).pin_memory().numpy()
    for c in (0, 4):
        assert np.array_equal(s.get_field(c), a[c // 4])
        assert np.array_equal(s.get_field(c, out=pinned), a[c // 4])
    assert not s.get_field(1).any()
    s.close()


def test_two_contexts_read_at_once():
    from dtmaxwell4_b200 import Simulation, abi
    n = (48, 150, 170)
    rng = np.random.default_rng(6)
    sims, want, got = [], [], [None, None]
    for q in range(2):
        s = Simulation(abi.make_config(*n, absorber=abi.ABS_NONE, pml=0))
        want.append(rng.standard_normal(n).astype(np.float32))
        s.set_field(2, want[q])
        sims.append(s)

    def read(q):
        for _ in range(8):
            got[q] = sims[q].get_field(2)
            if not np.array_equal(got[q], want[q]):
                return
    th = [threading.Thread(target=read, args=(q,)) for q in range(2)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    for q in range(2):
        assert np.array_equal(got[q], want[q])
        sims[q].close()


def test_spectra_are_complex_arrays():
    from dtmaxwell4_b200 import Simulation, abi
    n = (12, 150, 160)
    s = Simulation(abi.make_config(*n, absorber=abi.ABS_NONE, pml=0))
    om = [0.2, 0.3, 0.5, 0.7, 0.9, 1.1, 1.3, 1.5]
    d = s.add_dft_plane(0, 6, (1 << abi.EY) | (1 << abi.HZ), om)          # 6.1 MB
    f = np.random.default_rng(3).standard_normal(n).astype(np.float32)
    s.set_field(abi.EY, f)
    s.step(1)
    e = s.get_field(abi.EY)[6]
    out = s.read_dft(d)
    assert out.dtype == np.complex128 and out.shape == (2, len(om)) + n[1:]
    dt = s.cfg.dt
    for k, w in enumerate(om):
        assert np.allclose(out[0, k], e * np.exp(-1j * w * dt) * dt, rtol=0, atol=1e-12 * np.abs(e).max())
    s.close()


@pytest.mark.parametrize("n", [(9, 8, 11), (64, 161, 103), (128, 128, 64), (128, 128, 65)])
def test_without_memory_for_the_dense_copy(n):
    """No device memory for the dense copy of padded rows (kept by the context up to
    4 MB, from the stream's pool above): the strided copy gives the same."""
    from dtmaxwell4_b200 import Simulation, abi
    s = Simulation(abi.make_config(*n, absorber=abi.ABS_NONE, pml=0))
    a = np.random.default_rng(7).standard_normal(n).astype(np.float32)
    for k in range(2):                            # (then with it)
        s.fail_next(abi.FAIL_ALLOC, 0 if k == 0 else -1)
        s.set_field(4, a)
        s.fail_next(abi.FAIL_ALLOC, 0 if k == 0 else -1)
        assert np.array_equal(s.get_field(4), a)
        a = a + 1
    s.close()


def test_a_parked_context_keeps_no_dense_copy():
    import torch
    from dtmaxwell4_b200 import Simulation, abi
    n = (100, 100, 100)
    s = Simulation(abi.make_config(*n, absorber=abi.ABS_NONE, pml=0, parkable=True))
    a = np.random.default_rng(8).standard_normal(n).astype(np.float32)
    s.park()
    without = torch.cuda.mem_get_info()[0]
    s.unpark()
    s.set_field(4, a)
    s.park()
    assert torch.cuda.mem_get_info()[0] == without
    s.unpark()
    assert np.array_equal(s.get_field(4), a)
    s.close()


def test_cost_of_setting_a_small_field():
    """48^3 cells with padded rows: well below 250 us (a block from the pool on every
    call took 450, the strided copy takes 160)."""
    import time
    from dtmaxwell4_b200 import Simulation, abi
    s = Simulation(abi.make_config(48, 48, 48, pml=8))
    a = np.ones((48, 48, 48), np.float32)
    best = 1e9
    for _ in range(12):
        t = time.perf_counter()
        s.set_field(2, a)
        best = min(best, time.perf_counter() - t)
    assert best <= 250e-6, best
    s.close()

