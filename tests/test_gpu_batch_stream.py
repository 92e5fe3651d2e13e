"""A batch on a stream of its own, beside work on the default stream: its shared kernel's arguments, made
again whenever the graph is, reach it in order."""
import dataclasses

import numpy as np
import pytest

from abd_warp_b200 import scenes

pytestmark = pytest.mark.gpu


def test_batch_on_a_stream():
    import torch
    from abd_warp_b200.batch import BatchSimulator
    sc = [scenes.small_pile(1 + i % 3, 1 + i % 2, seed=i, level=1, plane=i % 4 == 0) for i in range(10)]
    prms = [p for _, p in sc]
    alone = BatchSimulator([b for b, _ in sc], prms)
    m = torch.zeros(1 << 24, device="cuda")
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        batch = BatchSimulator([b for b, _ in sc], prms)
    try:
        for step in range(12):
            ref = alone.step_sequential()
            for _ in range(50):
                m.add_(1.0)
            with torch.cuda.stream(stream):
                got = batch.step()
            for i, s in enumerate(batch.sims):
                for k in ("newton_iters", "linear_iters", "ls_trials", "n_active", "energy", "alpha"):
                    assert got[i][k] == ref[i][k], (step, i, k)
                np.testing.assert_array_equal(s.states.p0.cpu().numpy(), alone.sims[i].states.p0.cpu().numpy())
            if step % 3 == 2:  # other parameters: the graph and its arguments are made again
                prms = [dataclasses.replace(p, kappa=p.kappa * 1.25) for p in prms]
                for b in (batch, alone):
                    for s, p in zip(b.sims, prms):
                        s.set_params(p)
    finally:
        batch.close()
        alone.close()
