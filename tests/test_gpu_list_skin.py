"""The kept list's displacement where it grows: a list that an iteration asked for in mid-step makes the
next one's displacement larger, and two bodies that then approach each other by more than their own list's
displacement still meet, as in the oracle, bit for bit."""
import numpy as np
import pytest

import oracle
from abd_warp_b200 import scenes
from abd_warp_b200.params import SimParams

pytestmark = pytest.mark.gpu
KEYS = ("A0", "p0", "Adot", "pdot")
GAP = 0.023      # between the two bodies: the first list (8 dhat a body) does not hold their pairs,
SPEED = 0.16     # 1.6 mm a step each: they meet after 7 steps, 12 mm from where the list was made


def _scene(seed):
    """A sphere and a cube facing each other along x (unrotated, so that the list's boxes are tight), and far
    away the body that leaves its region."""
    y, z = np.random.default_rng(seed).uniform(-0.05, 0.05, size=2)
    bodies = [scenes._body("icosphere:3:0.2", (-0.5, 0.0, 0.0)), scenes._body("cube:0.3", (0.5, y, z)),
              scenes._body("cube:0.3", (9.0, 0.0, 0.0))]
    x = [b.V @ np.asarray(b.A) + np.asarray(b.p) for b in bodies]
    bodies[1].p = np.asarray(bodies[1].p, dtype=np.float64) - np.array([x[1][:, 0].min() - x[0][:, 0].max() - GAP, 0.0, 0.0])
    return bodies, SimParams(gravity=0.0, max_iter=1)


def _load(sims, o):
    import torch
    s = o.get_state()
    for sim in sims:
        for k in KEYS:
            getattr(sim.states, k).copy_(torch.as_tensor(s[k]))
        sim.dq = torch.as_tensor(np.asarray(s["dq"]).reshape(-1, 12))


@pytest.mark.parametrize("together", [1, 10])
@pytest.mark.parametrize("seed", [0, 1])
def test_approach_after_the_displacement_grew(seed, together):
    """together: alone, and as scenes of a batch that share a kernel."""
    from abd_warp_b200.batch import BatchSimulator
    from abd_warp_b200.simulator import AffineBodySimulator
    bodies, prm = _scene(seed)
    o = oracle.Oracle(scenes.flatten_bodies(bodies), prm)
    batch = BatchSimulator([_scene(seed)[0] for _ in range(together)], prm) if together > 1 else None
    sims = batch.sims if batch else [AffineBodySimulator(bodies=bodies, params=prm)]

    def step():
        r = o.step()
        for sim, i in zip(sims, batch.step() if batch else [sims[0].step()]):
            s = o.get_state()
            for k in ("newton_iters", "ls_trials", "n_pt", "n_ee", "n_ij", "n_active", "energy"):
                assert i[k] == r[k], k
            for k in KEYS:
                assert np.array_equal(getattr(sim.states, k).cpu().numpy(), s[k]), k
        return r

    # the far body moves by 30 mm a step while it stretches by 45 mm, which its orthogonality energy
    # resists: the step's one iteration goes neither to the predicted DOFs nor stays, and asks for a
    # list around it, from the iterate (the step's start) on
    s = o.get_state()
    A, p, zA, zp = np.array(s["A0"]), np.array(s["p0"]), np.zeros((3, 3, 3)), np.zeros((3, 3))
    W, v = zA.copy(), zp.copy()
    W[2, 0, 0], v[2, 0] = 30.0, 3.0
    o.set_state(A, p, W, v, dq=np.zeros((3, 12)))
    _load(sims, o)
    step()
    # it is put back, at rest; the other two approach each other
    v = zp.copy()
    v[0, 0], v[1, 0] = SPEED, -SPEED
    o.set_state(A, p, zA, v, dq=np.zeros((3, 12)))
    _load(sims, o)
    met = sum(step()["n_pt"] > 0 for _ in range(14))
    assert met > 0
