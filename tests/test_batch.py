"""Batched forward + adjoint of independent instances of uneven sizes: the
interleaved batch returns exactly what separate runs return."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _make(sc):
    from dtmaxwell4_b200 import Simulation, scenarios
    s = Simulation(sc["cfg"])
    scenarios.apply(s, sc)
    s.set_design(*sc["design"])
    return s


@pytest.mark.parametrize("budget", [-1, 0])
def test_batch_equals_separate_runs(budget):
    """budget -1: recorded design histories; 0: checkpointed recompute in the batch."""
    from dtmaxwell4_b200 import engine, scenarios
    scs = [scenarios.design_block_instance(seed, edges=(40, 48, 56, 64), pml=6, design=6, steps=48, nblocks=3)
           for seed in range(5)]
    shapes = {(sc["cfg"].nx, sc["cfg"].ny, sc["cfg"].nz) for sc in scs}
    assert len(shapes) > 1
    sims = [_make(sc) for sc in scs]
    for s in sims:
        s.set_adjoint_memory(budget)
    J, G = engine.batch_forward_adjoint(sims, 48, [sc["plane_x"] for sc in scs], [sc["omega"] for sc in scs],
                                        checkpoint_every=20)
    for b, sc in enumerate(scs):
        s = _make(sc)
        Jb, gb = s.forward_adjoint(48, sc["plane_x"], sc["omega"], 20)
        assert J[b] == Jb and np.array_equal(G[b], gb), b
        for c in range(6):
            assert np.array_equal(s.get_field(c), sims[b].get_field(c))
        s.close()
        sims[b].close()


def test_cost_of_a_first_batch():
    """The first batch on new contexts takes at most three of a later one (four to five
    where the pool passed blocks between streams in flight)."""
    import time
    from dtmaxwell4_b200 import Simulation, abi, engine
    n, best = (64, 64, 64), 1e9
    for _ in range(4):
        sims = []
        for q in range(8):
            s = Simulation(abi.make_config(*n, courant=0.4, pml=6))
            s.set_design((32, 32, 32), np.full((3, 6, 6, 6), 2.0, np.float32))
            s.set_field(2, np.random.default_rng(q).standard_normal(n).astype(np.float32))
            sims.append(s)
        t = []
        for _ in range(3):
            a = time.perf_counter()
            engine.batch_forward_adjoint(sims, 30, [54] * 8, [0.4] * 8)
            t.append(time.perf_counter() - a)
        best = min(best, t[0] / min(t[1:]))
        for s in sims:
            s.close()
    assert best <= 3.0, best
