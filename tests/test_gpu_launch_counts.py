"""The launch counts of a scene stepped alone and in a batch, in turn: each step counts its own graph's
kernels, whatever was captured in between."""
import pytest

from abd_warp_b200 import scenes

pytestmark = pytest.mark.gpu
KEYS = ("A0", "p0", "Adot", "pdot")


# 3 scenes: a branch each; 9 scenes: a shared kernel
@pytest.mark.parametrize("together", [3, 9])
def test_alone_and_in_a_batch(together):
    from abd_warp_b200.batch import BatchSimulator
    batch = BatchSimulator([scenes.small_pile(2, 1, seed=i, level=0)[0] for i in range(together)])
    sim = batch.sims[0]
    try:
        for _ in range(2):  # (free fall)
            batch.step_sequential()
        saved = [getattr(sim.states, k).clone() for k in KEYS] + [sim.dq]

        def count(step):
            for k, v in zip(KEYS, saved):
                getattr(sim.states, k).copy_(v)
            sim.dq = saved[-1]
            sim.collision_set_dofs(sim.states.A0, sim.states.p0)  # (the step makes its candidate list)
            n = sim.launch_count()
            step()
            return sim.launch_count() - n

        alone, shared = count(sim.step), count(batch.step)
        assert alone > 0 and shared > 0
        for _ in range(2):
            assert count(sim.step) == alone
            assert count(batch.step) == shared
            assert count(batch.step) == shared
            assert count(sim.step) == alone
    finally:
        batch.close()
