"""The solve kernel's start: its clusters of CTAs begin while other work holds the SMs, so that a
cluster's CTAs start apart; every solve gives the bits of a solve on an idle GPU."""
import pytest

from abd_warp_b200 import scenes

pytestmark = pytest.mark.gpu


# bodies (ground box included) 17, 65, 257: clusters of 2, 8 and 16 CTAs
@pytest.mark.parametrize("solver", [0, 1])
@pytest.mark.parametrize("side,layers", [(4, 1), (4, 4), (8, 4)])
def test_solve_beside_other_work(side, layers, solver):
    import torch
    from abd_warp_b200.simulator import AffineBodySimulator
    bodies, prm = scenes.small_pile(side, layers, seed=11, level=0, radius=0.2)
    prm.solver = solver
    sim = AffineBodySimulator(bodies=bodies, params=prm)
    for _ in range(16):
        sim.step()
    sim.gradient_hessian(sim.states.A0, sim.states.p0)
    dq0 = torch.full((len(bodies), 12), 1e-3, dtype=torch.float64, device="cuda")
    want, it = sim.solve(dq0)
    busy, done = torch.cuda.Stream(), torch.cuda.Event()
    m = torch.zeros(1 << 22, device="cuda")
    for k in range(40):
        with torch.cuda.stream(busy):
            for _ in range(4):
                m.add_(1.0)
            done.record()
        got, n = sim.solve(dq0)
        assert n == it and torch.equal(got, want)
    busy.synchronize()
