"""Calls that were refused device memory, and the calls after them.

dtmx_fail_next refuses one allocation after another on the host, as if the
memory were not there.  A call then either does without (the automatic
engine's second set of fields, the single-sweep adjoint's second psi: the same result,
bit for bit) or reports DTMX_ERR_OOM, and the same call afterwards, from the
same state, gives what it gives on a context that was never refused any.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = (20, 18, 21)
OMEGA = 0.4


def _sim(engine):
    from dtmaxwell4_b200 import Simulation, abi
    # no absorber: the six fields are the whole state
    s = Simulation(abi.make_config(*N, courant=0.5, absorber=abi.ABS_NONE, pml=0))
    rng = np.random.default_rng(3)
    s.set_design((6, 5, 7), rng.uniform(1.0, 4.0, size=(3, 4, 5, 6)).astype(np.float32))
    s.set_engine(engine)
    return s


def _fields(s):
    rng = np.random.default_rng(5)
    for c in range(6):
        s.set_field(c, rng.standard_normal(N).astype(np.float32))


def _gradient(s, history):
    s.set_adjoint_memory(-1 if history else 0)
    return s.forward_adjoint(12, 15, OMEGA, 5)


@pytest.mark.parametrize("engine", [0, 1])
@pytest.mark.parametrize("history", [True, False])
def test_gradient_after_a_refused_allocation(engine, history):
    from dtmaxwell4_b200 import abi
    from dtmaxwell4_b200.engine import DtmxError
    s = _sim(engine)
    _fields(s)
    # by the step the run starts from: the objective's phases round differently
    want = {0: _gradient(s, history)}
    _fields(s)
    want[12] = _gradient(s, history)
    assert len(want) == 2 and all(J != 0.0 and np.abs(g).max() > 0 for J, g in want.values())
    s.close()
    refused = 0
    for k in range(48):
        s = _sim(engine)
        _fields(s)
        s.fail_next(abi.FAIL_ALLOC, k)
        try:
            first = _gradient(s, history)
        except DtmxError as e:
            assert e.code == abi.ERR_OOM
            refused += 1
        else:
            assert first[0] == want[0][0] and np.array_equal(first[1], want[0][1]), k
        s.fail_next(abi.FAIL_ALLOC, -1)
        _fields(s)
        J, grad = want[s.nstep]
        again = _gradient(s, history)
        assert again[0] == J and np.array_equal(again[1], grad), k
        s.close()
    assert refused >= 8              # the objective's four arrays and three tables, the history or the checkpoints
