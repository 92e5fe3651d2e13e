"""Solves at the size where the solve changes its kernels: systems that one cluster holds and
systems that the whole-GPU kernels take, alone and inside the device loop, against the oracle, bit for bit."""
import dataclasses

import numpy as np
import pytest

import oracle
from abd_warp_b200 import scenes

pytestmark = pytest.mark.gpu
KEYS = ("A0", "p0", "Adot", "pdot")


def _scene(side, layers, plane, warm, **kw):
    """A new simulator and an oracle in the state of another one after `warm` steps."""
    from abd_warp_b200.simulator import AffineBodySimulator
    bodies, prm = scenes.small_pile(side, layers, seed=3, level=0, plane=plane)
    first = AffineBodySimulator(bodies=bodies, params=prm)
    for _ in range(warm):
        first.step()
    prm = dataclasses.replace(prm, **kw)
    sim = AffineBodySimulator(bodies=bodies, params=prm)
    for k in KEYS:
        getattr(sim.states, k).copy_(getattr(first.states, k))
    sim.dq = first.dq
    o = oracle.Oracle(scenes.flatten_bodies(bodies), prm)
    s = {k: getattr(sim.states, k).cpu().numpy() for k in KEYS}
    o.set_state(*[s[k] for k in KEYS], dq=sim.dq.cpu().numpy())
    first.close()
    return sim, o, s


# 4,096 bodies: the cluster kernel; more: the large one, with clusters of one body and of several
@pytest.mark.parametrize("solver", [0, 1])
@pytest.mark.parametrize("side,layers,plane,warm,precond", [(64, 1, True, 24, 0), (64, 1, False, 24, 0), (45, 4, False, 60, 0),
                                                            (45, 4, False, 60, 1), (56, 4, False, 45, 1)])
def test_solve(side, layers, plane, warm, precond, solver):
    import torch
    sim, o, s = _scene(side, layers, plane, warm, precond=precond, solver=solver, cg_max_iter=30)
    A, p = (torch.as_tensor(s[k], device="cuda") for k in ("A0", "p0"))
    got = sim.gradient_hessian(A, p)
    ref = o.gh(s["A0"], s["p0"])
    assert np.array_equal(got["g"].cpu().numpy(), np.asarray(ref["g"]).reshape(got["g"].shape))
    dq0 = np.random.default_rng(5).normal(0.0, 1e-3, size=(sim.n_bodies, 12))
    want, it = o.solve(dq0)
    for _ in range(2):
        dq, n = sim.solve(torch.as_tensor(dq0, device="cuda"))
        assert n == it
        assert np.array_equal(dq.cpu().numpy(), np.asarray(want).reshape(-1, 12))


# (tiny: lists that overflow, so that iterations and solves are skipped)
@pytest.mark.parametrize("solver", [0, 1])
@pytest.mark.parametrize("loop,tiny", [(0, 0), (0, 64), (1, 0)])
def test_steps(loop, tiny, solver):
    sim, o, _ = _scene(64, 1, False, 22, precond=0, solver=solver, newton_loop=loop, min_capacity=tiny, max_iter=4)
    active = 0
    for _ in range(3):
        i, r = sim.step(), o.step()
        s = o.get_state()
        for k in KEYS:
            assert np.array_equal(getattr(sim.states, k).cpu().numpy(), s[k]), k
        for k in ("newton_iters", "linear_iters", "ls_trials", "n_pt", "n_ee", "n_ij", "n_active", "energy"):
            assert i[k] == r[k], k
        active += i["n_active"]
    assert active > 0


def test_in_a_batch():
    from abd_warp_b200.batch import BatchSimulator
    sc = [scenes.small_pile(64, 1, seed=3, level=0), scenes.small_pile(2, 2, seed=4, level=0)]
    batch, alone = (BatchSimulator([b for b, _ in sc], [p for _, p in sc]) for _ in range(2))
    try:
        for _ in range(24):
            got, ref = batch.step(), alone.step_sequential()
            for g, r in zip(got, ref):
                assert {k: v for k, v in g.items()} == {k: v for k, v in r.items()}
            for a, b in zip(batch.sims, alone.sims):
                assert np.array_equal(a.states.p0.cpu().numpy(), b.states.p0.cpu().numpy())
    finally:
        batch.close()
        alone.close()
