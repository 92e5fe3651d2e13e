"""The kept list with barrier distances that are not small against the bodies: the same bits as the
oracle, and no more memory than a list of the most candidates that its rule lets grow, its
line-search copy and half as much again (2 x 1.5 x 2^20 x 16 B = 48 MB; the bound leaves room for
the other lists)."""
import dataclasses

import numpy as np
import pytest

import oracle
from abd_warp_b200 import scenes

pytestmark = pytest.mark.gpu
KEYS = ("A0", "p0", "Adot", "pdot")


@pytest.mark.parametrize("level,dhat,full", [(3, 0.05, 0), (3, 0.05, 1), (2, 0.1, 0), (1, 0.3, 0)])
def test_large_barrier_distance(level, dhat, full):
    import torch
    from abd_warp_b200.simulator import AffineBodySimulator
    bodies, prm = scenes.small_pile(2, 2, seed=3, level=level)
    prm = dataclasses.replace(prm, dhat=dhat, ipc_full=full)
    o = oracle.Oracle(scenes.flatten_bodies(bodies), prm)
    sim = AffineBodySimulator(bodies=bodies, params=prm)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    active = 0
    for _ in range(10):
        i, r = sim.step(), o.step()
        s = o.get_state()
        for k in KEYS:
            assert np.array_equal(getattr(sim.states, k).cpu().numpy(), s[k]), k
        for k in ("newton_iters", "linear_iters", "ls_trials", "n_pt", "n_ee", "n_ij", "n_active", "energy"):
            assert i[k] == r[k], k
        active += i["n_active"]
    assert active > 0
    assert free - torch.cuda.mem_get_info()[0] < 128 << 20
