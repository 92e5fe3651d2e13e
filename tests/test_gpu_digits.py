"""The bodies' exact sums with many folds of their counters: a body of 655,362 vertices on the ground
plane (20 folds; its vertex-ground gradient is negative) against the oracle, bit for bit."""
import numpy as np
import pytest

import oracle
from abd_warp_b200 import scenes
from abd_warp_b200.affine_body import AffineMesh
from abd_warp_b200.params import SimParams

pytestmark = pytest.mark.gpu


def test_large_body_on_the_plane():
    import torch
    from abd_warp_b200.simulator import AffineBodySimulator
    prm = SimParams(ground_enabled=True, ground=0.0, max_iter=2)
    y = 0.2 + 0.3 * prm.dhat  # (its lowest vertices lie within dhat)
    bodies = [scenes._body("icosphere:8:0.2", (0.0, y, 0.0))]
    flat = scenes.flatten_bodies(bodies)
    o = oracle.Oracle(flat, prm)
    sim = AffineBodySimulator(bodies=bodies, params=prm)
    got, ref = sim.gradient_hessian(sim.states.A0, sim.states.p0), o.gh(flat["A"], flat["p"])
    assert np.array_equal(got["g"].cpu().numpy(), np.asarray(ref["g"]).reshape(1, 12))
    assert np.array_equal(got["diag"].cpu().numpy(), np.asarray(ref["diag"]).reshape(1, 12, 12))
    i, r = sim.step(), o.step()
    assert i["n_vg"] == r["n_vg"] > 0 and i["energy"] == r["energy"]
    s = o.get_state()
    for k in ("A0", "p0", "Adot", "pdot"):
        assert np.array_equal(getattr(sim.states, k).cpu().numpy(), s[k]), k
