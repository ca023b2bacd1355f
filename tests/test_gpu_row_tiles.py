"""The row-shaped passes on grids of fewer full tiles than SMs: one row per block with a thread
per cell, several rows, and rows longer than a block, single and batched, against the FP64
oracle's trajectory."""
import numpy as np
import pytest

from helpers import rand_m, to_np

pytestmark = pytest.mark.gpu


# one row per block with a thread per cell, several rows, and rows longer than a block
@pytest.mark.parametrize("n", [(1, 2, 64), (1, 3, 8), (1, 33, 16), (1, 128, 128), (1, 40, 512), (2, 5, 1024),
                               (1, 38, 96), (3, 11, 150)])
@pytest.mark.parametrize("nsim", [1, 3])
def test_small_grid_steps_match_oracle(n, nsim):
    """Batched: every simulation with its own material, field, mask and state, so that a row, a
    scalar or a spectrum taken from another one shows."""
    import oracle as O
    from mumax2 import Plan
    prob = O.full_desc(n=n, cell=(3e-9, 4e-9, 4e-9), demag=1, exchange=1, zeeman=1, msat=8e5, aex=1.3e-11, alpha=0.1,
                       bext=(0.0, 0.01, 0.02), demag_accuracy=2)
    N = n[0] * n[1] * n[2]
    sims, masks, states = [], [], []
    for b in range(nsim):
        sims.append(dict(prob, msat=8e5 - 1.5e5 * b, alpha=0.1 + 0.2 * b, bext=(0.01 * b, 0.01, 0.02 - 0.01 * b)))
        masks.append((np.arange(N) % (7 + b) != 3).astype(np.float32))
        states.append(rand_m(n, seed=9 + b) * np.tile(masks[b], 3))
    if nsim > 1:
        g = Plan(prob, masks={"msat": np.concatenate(masks)}, sims=sims, masks_per_sim=True)
    else:
        g = Plan(prob, masks={"msat": masks[0]})
    g.solver("rk23", dt=1e-14, maxerr=1e-5)
    g.set_state(np.concatenate(states))
    g.steps(3)
    got = to_np(g.get_state()).reshape(nsim, -1)
    for b in range(nsim):
        r = O.OracleRun(O.Oracle(dict(sims[b], masks={"msat": masks[b]})), states[b], solver="rk23", dt=1e-14,
                        maxerr=1e-5)
        for _ in range(3):
            r.step()
        assert np.abs(got[b] - r.m).max() < 2e-5   # the trajectory bar of a few steps
    g.close()
