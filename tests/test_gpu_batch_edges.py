"""The batch's shared kernel at the edges of what it takes (192 bodies and one more; 65,536 vertices and
edges and more): each scene has the result of its own steps, bit for bit."""
import numpy as np
import pytest

from abd_warp_b200 import scenes

pytestmark = pytest.mark.gpu


# (side, layers, level, plane): 192 bodies on the plane, 193 with the ground box, 41,000 and 164,000
# vertices and edges, among small scenes
@pytest.mark.parametrize("large", [[(8, 3, 0, True)], [(8, 3, 0, False)], [(2, 2, 4, False)], [(2, 2, 5, False)],
                                   [(8, 3, 0, True), (2, 2, 4, False), (2, 4, 4, False)]])
def test_edges(large):
    from abd_warp_b200.batch import BatchSimulator
    sc = [scenes.small_pile(s, l, seed=5, level=v, plane=p) for s, l, v, p in large]
    sc += [scenes.small_pile(1 + i % 3, 1 + i % 2, seed=i, level=1) for i in range(11)]
    batch, alone = (BatchSimulator([b for b, _ in sc], [p for _, p in sc]) for _ in range(2))
    seen = 0
    try:
        for step in range(22):
            got, ref = batch.step(), alone.step_sequential()
            for i, (g, r) in enumerate(zip(got, ref)):
                assert g == r, (step, i)
                for k in ("A0", "p0", "Adot", "pdot"):
                    np.testing.assert_array_equal(getattr(batch.sims[i].states, k).cpu().numpy(),
                                                  getattr(alone.sims[i].states, k).cpu().numpy())
            seen += sum(g["n_active"] + g["n_vg"] for g in got[:len(large)])
        assert seen > 0
    finally:
        batch.close()
        alone.close()
