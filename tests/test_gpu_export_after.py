"""The system exported (and solved) after a step when other calls came between: a culling that renumbers
the pair arrays, changed parameters.  With one Newton iteration the step's system is the one at
its start, which the oracle assembles."""
import ctypes
import dataclasses

import numpy as np
import pytest

import oracle
from abd_warp_b200 import _lib, scenes

pytestmark = pytest.mark.gpu
KEYS = ("A0", "p0", "Adot", "pdot")


def _pair(**kw):
    import torch
    from abd_warp_b200.simulator import AffineBodySimulator
    bodies, prm = scenes.small_pile(2, 2, seed=21, level=1, radius=0.2)
    prm = dataclasses.replace(prm, max_iter=1, **kw)
    o = oracle.Oracle(scenes.flatten_bodies(bodies), prm)
    sim = AffineBodySimulator(bodies=bodies, params=prm)
    for _ in range(24):
        o.step()
    s = o.get_state()
    for k in KEYS:
        getattr(sim.states, k).copy_(torch.as_tensor(s[k]))
    sim.dq = torch.as_tensor(np.asarray(s["dq"]).reshape(-1, 12))
    return sim, o, prm


def _export(sim):
    import torch
    n, m = sim.n_bodies, ctypes.c_int(0)
    g = torch.zeros((n, 12), dtype=torch.float64, device="cuda")
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    _lib.check(sim._L.abd_export_system(sim._h, p(g), None, None, None, 0, ctypes.byref(m)), "export")
    off = torch.zeros((max(m.value, 1), 12, 12), dtype=torch.float64, device="cuda")
    ij = torch.zeros((max(m.value, 1), 2), dtype=torch.int32, device="cuda")
    _lib.check(sim._L.abd_export_system(sim._h, None, None, p(off), p(ij), m.value, ctypes.byref(m)), "export")
    return g.cpu().numpy(), off[:m.value].cpu().numpy(), ij[:m.value].cpu().numpy()


def _step(sim, o, prm):
    import torch
    s = o.get_state()
    A, p = np.array(s["A0"]), np.array(s["p0"])
    ref = o.gh(A, p)
    dq0 = np.full((sim.n_bodies, 12), 1e-3)
    solved = (dq0, *o.solve(dq0))
    # (a culling clears the list of coupled pairs: a solve after it has clusters of one body)
    o.set_params(dataclasses.replace(prm, precond=0))
    alone = (dq0, *o.solve(dq0))
    o.set_params(prm)
    o.set_state(*[s[k] for k in KEYS], dq=s["dq"])  # (solve leaves its solution as the warm start)
    sim.step()
    o.step()
    return torch.as_tensor(A, device="cuda"), torch.as_tensor(p, device="cuda"), ref, solved, alone


def _same_system(sim, ref, solved):
    import torch
    g, off, ij = _export(sim)
    assert np.array_equal(ij, ref["ij"])
    assert np.array_equal(off, np.asarray(ref["off"]).reshape(-1, 12, 12))
    assert np.array_equal(g, np.asarray(ref["g"]).reshape(g.shape))
    dq0, x, it = solved
    got, n = sim.solve(torch.as_tensor(dq0, device="cuda"))
    assert n == it and np.array_equal(got.cpu().numpy(), np.asarray(x).reshape(-1, 12))


def _same_state(sim, o):
    s = o.get_state()
    for k in KEYS:
        assert np.array_equal(getattr(sim.states, k).cpu().numpy(), s[k]), k


@pytest.mark.parametrize("before", [False, True])
def test_culling_at_the_same_dofs(before):
    """before: the system is also exported before the culling."""
    sim, o, prm = _pair()
    blocks = 0
    for _ in range(3):
        A, p, ref, solved, alone = _step(sim, o, prm)
        if before:
            _same_system(sim, ref, solved)
        sim.collision_set_dofs(A, p)
        _same_system(sim, ref, alone)
        _same_state(sim, o)
        blocks += int((np.abs(np.asarray(ref["off"])) > 0).any())
    assert blocks > 0


@pytest.mark.parametrize("scenes_together", [1, 10])
def test_solve_after_a_step(scenes_together):
    """A solve of the step's last system has the pass's preconditioner clusters: alone and in a batch whose
    scenes share a kernel."""
    import torch
    from abd_warp_b200.batch import BatchSimulator
    sim, o, prm = _pair()
    sims = [sim]
    if scenes_together > 1:
        batch = BatchSimulator([scenes.small_pile(2, 2, seed=21, level=1, radius=0.2)[0] for _ in range(scenes_together)], prm)
        sims = batch.sims
        for s in sims:
            for k in KEYS:
                getattr(s.states, k).copy_(getattr(sim.states, k))
            s.dq = sim.dq
    for _ in range(2):
        s = o.get_state()
        o.gh(s["A0"], s["p0"])
        dq0 = np.full((sim.n_bodies, 12), 1e-3)
        want, it = o.solve(dq0)
        o.set_state(*[s[k] for k in KEYS], dq=s["dq"])
        o.step()
        if scenes_together > 1:
            batch.step()
        else:
            sim.step()
        for s in sims:
            got, n = s.solve(torch.as_tensor(dq0, device="cuda"))
            assert n == it and np.array_equal(got.cpu().numpy(), np.asarray(want).reshape(-1, 12))


@pytest.mark.parametrize("call", ["static", "swept", "positions"])
def test_culling_elsewhere(call):
    """The pair list is then that culling's; the export stays inside its buffers and the step after it is
    right."""
    sim, o, prm = _pair()
    for _ in range(3):
        _step(sim, o, prm)
        s = sim.states
        if call == "static":
            ij = sim.collision_set_dofs(s.A0, s.p0 * 0.25)[0]  # (bodies drawn together: more pairs)
        elif call == "swept":
            ij = sim.collision_set_dofs(s.A0, s.p0, s.A0, s.p0 * 0.25)[0]
        else:
            ij = sim.collision_set(sim.transform(s.A0, s.p0 * 0.25))[0]
        got = _export(sim)[2]
        assert np.array_equal(got, ij.cpu().numpy()) and len(got) > 0
        _same_state(sim, o)


@pytest.mark.parametrize("change", [{"dhat": 4e-3}, {"dhat": 1e-4}, {"friction_mu": 0.0}, {"friction_mu": 0.4}])
def test_parameters_changed_before_the_export(change):
    """The pairs are those of the parameters the system was made with."""
    mu = "friction_mu" in change
    kw = dict(ipc_full=1, friction_mu=0.2) if mu else {}
    sim, o, prm = _pair(**kw)
    twin, _, _ = _pair(**kw)
    for _ in range(2):
        sim.step()
        twin.step()
        want = _export(twin)
        sim.set_params(dataclasses.replace(prm, **change))
        for a, b in zip(_export(sim), want):
            assert np.array_equal(a, b)
        sim.set_params(prm)
