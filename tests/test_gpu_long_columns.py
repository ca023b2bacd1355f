"""Columns of 600 to 2048 rows, at every number of columns that a block takes, masked, periodic
and batched, and z axes whose multiply is not in registers: the demag field against the
convolution with the plan's own kernel in FP64 (torch)."""
import numpy as np
import pytest

from helpers import rand_m, rel_err, to_np

pytestmark = pytest.mark.gpu


def _prob(n, pbc=(0, 0, 0)):
    return dict(n=n, cell=(3e-9, 4e-9, 5e-9), pbc=pbc, demag=1, exchange=1, msat=8e5, aex=1.3e-11, alpha=0.05,
                demag_accuracy=1)


def _field64(plan, n, pbc, m, mask, msat):
    """Ms irfft(K rfft(mask m)) in FP64.  The stored octant of K (xx yy zz yz xz xy) is even along
    every axis but odd along s and d for K_sd."""
    import torch
    L = [s if s == 1 or p else 2 * s for s, p in zip(n, pbc)]
    k = torch.from_numpy(plan.demag_kernel()).cuda().double()
    at = [torch.arange(v, device="cuda") for v in (L[0], L[1], L[2] // 2 + 1)]
    neg = [1.0 - 2.0 * (a > v // 2) for a, v in zip(at, L)]
    fold = [torch.where(a > v // 2, v - a, a) for a, v in zip(at, L)]
    k = k[:, fold[0]][:, :, fold[1]]
    sign = {3: neg[1][None, :, None], 4: neg[0][:, None, None], 5: neg[0][:, None, None] * neg[1][None, :, None]}
    for q, s in sign.items():
        k[q] *= s
    v = (torch.from_numpy(m.reshape(3, -1)).cuda().double() * torch.from_numpy(mask).cuda().double()).reshape(3, *n)
    f = torch.fft.rfftn(v, s=L, dim=(1, 2, 3))
    h = torch.stack([k[0] * f[0] + k[5] * f[1] + k[4] * f[2], k[5] * f[0] + k[1] * f[1] + k[3] * f[2],
                     k[4] * f[0] + k[3] * f[1] + k[2] * f[2]])
    h = torch.fft.irfftn(h, s=L, dim=(1, 2, 3), norm="forward")[:, :n[0], :n[1], :n[2]]
    return to_np(msat * h).ravel()


# 2048-point columns by parity, two and four columns to a block (a ragged last one); columns of up
# to 4096 points, one, two and four; periodic axes; two layers; z axes of 18 to 256 layers, in
# columns and in the four-step pass, padded and periodic.  FP32 transforms of up to 4096 points:
# eps * log2(L) each way, as in test_gpu_sizes
@pytest.mark.parametrize("n,pbc", [((1, 1024, 4), (0, 0, 0)), ((1, 1024, 256), (0, 0, 0)), ((1, 1024, 300), (0, 0, 0)),
                                   ((1, 700, 5), (0, 0, 0)), ((1, 600, 150), (0, 0, 0)), ((1, 600, 320), (0, 0, 0)),
                                   ((1, 1000, 1024), (0, 0, 0)), ((1, 1200, 6), (0, 0, 0)), ((1, 1300, 150), (0, 0, 0)),
                                   ((1, 2048, 4), (0, 0, 0)), ((1, 2048, 75), (0, 0, 0)), ((1, 2000, 192), (0, 0, 0)),
                                   ((1, 2048, 6), (0, 1, 0)), ((1, 1024, 8), (0, 1, 0)), ((2, 1024, 8), (0, 0, 0)),
                                   ((3, 1200, 6), (0, 0, 0)),
                                   ((4, 1024, 32), (0, 0, 0)), ((2, 2048, 5), (0, 0, 0)), ((2, 2048, 32), (0, 0, 0)),
                                   ((2, 2048, 6), (0, 1, 0)), ((2, 4096, 5), (1, 1, 0)), ((1, 4096, 6), (0, 1, 0)),
                                   ((1, 4096, 150), (0, 1, 0)), ((1, 2048, 150), (0, 1, 0)), ((32, 24, 30), (0, 0, 0)), ((128, 6, 10), (0, 0, 0)),
                                   ((256, 4, 6), (0, 0, 0)), ((8, 20, 12), (1, 0, 0)), ((16, 12, 20), (1, 0, 0)),
                                   ((64, 6, 8), (1, 1, 0)), ((18, 30, 40), (0, 0, 0)), ((20, 8, 6), (1, 0, 1))])
def test_field(n, pbc):
    from mumax2 import Plan
    mask = np.random.default_rng(n[2]).uniform(0.4, 1.0, n[0] * n[1] * n[2]).astype(np.float32)
    g = Plan(_prob(n, pbc), masks={"msat": mask})
    m = rand_m(n, seed=sum(n)).astype(np.float32)
    assert rel_err(to_np(g.fields(m)["demag"]), _field64(g, n, pbc, m, mask, 8e5)) < 1e-6
    g.close()


@pytest.mark.parametrize("n,along_y", [((1, 1024, 8), 0), ((1, 1024, 75), 0), ((1, 1200, 8), 0), ((4, 128, 128), 0), ((3, 100, 121), 0),
                                   ((1, 2048, 6), 1), ((2, 2048, 4), 1)])
def test_batched(n, along_y):
    """Every simulation of a batch with its own material, mask and state.  The bodies fill the GPU,
    so a block of their z multiply does several simulations, the last one fewer."""
    from mumax2 import Plan
    N, sims, pbc = n[0] * n[1] * n[2], 21, (0, along_y, 0)
    prob = _prob(n, pbc)
    msat = [8e5 * (1 - 0.02 * b) for b in range(sims)]
    masks = [np.random.default_rng(b).uniform(0.4, 1.0, N).astype(np.float32) for b in range(sims)]
    states = [rand_m(n, seed=b).astype(np.float32) for b in range(sims)]
    g = Plan(prob, masks={"msat": np.concatenate(masks)}, sims=[dict(prob, msat=v) for v in msat], masks_per_sim=True)
    got = to_np(g.fields(np.concatenate(states))["demag"]).reshape(sims, 3 * N)
    for b in range(sims):
        assert rel_err(got[b], _field64(g, n, pbc, states[b], masks[b], msat[b])) < 1e-6
    g.close()


def test_finished_simulations_in_a_group():
    """A block of the z multiply that does several simulations passes over those that have
    finished: each one's steps and state are those of its own plan."""
    from mumax2 import Plan
    n, sims = (4, 128, 128), 18
    prob = _prob(n)
    thr = np.where(np.arange(sims) % 3 == 1, 1e15, 1e-3)   # every third one stops at once
    msat = [8e5 * (1 - 0.02 * b) for b in range(sims)]
    states = [rand_m(n, seed=b).astype(np.float32) for b in range(sims)]
    g = Plan(prob, sims=[dict(prob, msat=v) for v in msat])
    g.solver("rk23", dt=1e-15, maxerr=1e-5)
    g.set_state(np.concatenate(states))
    g.batch_run_until_maxtorque(thr, max_steps=5)
    got, stats = g.get_state().reshape(sims, -1), g.batch_stats()
    assert len({s["step"] for s in stats}) == 2
    for b in range(0, sims, 5):
        one = Plan(dict(prob, msat=msat[b]))
        one.solver("rk23", dt=1e-15, maxerr=1e-5)
        one.set_state(states[b])
        one.run_until_maxtorque(thr[b], max_steps=5)
        assert one.stats()["step"] == stats[b]["step"]
        assert np.abs(got[b] - one.get_state()).max() < 2e-6   # rounding of the scaled spectrum, a few steps
        one.close()
    g.close()
