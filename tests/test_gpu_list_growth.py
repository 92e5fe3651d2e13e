"""Lists that outgrow their capacity while a step's iterations make their displacement larger: the step ends,
with the host loop's result (which keeps no list), bit for bit."""
import dataclasses

import numpy as np
import pytest

from abd_warp_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("level,seed", [(5, 16), (5, 22), (4, 3)])
def test_fine_meshes(level, seed):
    from abd_warp_b200.simulator import AffineBodySimulator
    bodies, prm = scenes.small_pile(2, 2, seed=seed, level=level)
    sims = [AffineBodySimulator(bodies=bodies, params=dataclasses.replace(prm, newton_loop=k)) for k in (0, 1)]
    for _ in range(14):
        a, b = (s.step() for s in sims)
        for k in ("newton_iters", "linear_iters", "ls_trials", "n_pt", "n_ee", "n_ij", "n_active", "energy", "alpha", "toi"):
            assert a[k] == b[k], k
        for k in ("A0", "p0", "Adot", "pdot"):
            assert np.array_equal(*(getattr(s.states, k).cpu().numpy() for s in sims)), k
