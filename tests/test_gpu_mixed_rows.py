"""Row output of the mixed-radix epilogue and stage combine: trajectories bit-identical to
separate row passes, on odd and even row lengths, films and bodies, masked, periodic and
batched."""
import numpy as np
import pytest

from helpers import rand_m
from test_gpu_epi_r2c import _compare

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,pbc", [((1, 15, 21), (0, 0, 0)), ((3, 20, 28), (0, 0, 0)), ((1, 16, 96), (0, 0, 0)),
                                   ((2, 9, 75), (0, 0, 0)), ((1, 12, 34), (0, 0, 0)), ((1, 10, 24), (0, 0, 1)),
                                   ((2, 7, 320), (0, 0, 0))])
@pytest.mark.parametrize("solver", ["rk23", "rk12"])
def test_row_output_bit_identical(monkeypatch, n, pbc, solver):
    import oracle as O
    mask = np.random.default_rng(2).uniform(0.4, 1.0, size=n[0] * n[1] * n[2]).astype(np.float32)
    prob = O.full_desc(n=n, cell=(2e-9, 4e-9, 4e-9), pbc=pbc, demag=1, exchange=1, zeeman=1, msat=9e5, aex=1.3e-11,
                       bext=(0.01, 0.0, 0.02), alpha=0.05, demag_accuracy=2)
    _compare(monkeypatch, prob, rand_m(n, seed=11), solver, 12, dt=1e-13, maxerr=1e-5)
    _compare(monkeypatch, dict(prob, masks={"msat": mask}), rand_m(n, seed=12), solver, 8, masks={"msat": mask},
             dt=1e-13, maxerr=1e-5)


def test_row_output_batched(monkeypatch):
    from mumax2 import workloads as W
    n = (3, 10, 12)
    prob = dict(n=n, cell=(2e-9, 4e-9, 4e-9), demag=1, exchange=1, anis=1, zeeman=1, msat=8e5, aex=1.3e-11, ku=2e5,
                anisu=(0.0, 0.6, 0.8), alpha=0.5, bext=(0.0, 0.01, 0.02), demag_accuracy=2)
    _, sims, _ = W.relax_set(5, seed=3)
    m0 = np.concatenate([rand_m(n, seed=s) for s in range(5)])
    _compare(monkeypatch, prob, m0, "rk23", 10, sims=sims, dt=1e-14, maxerr=1e-5)


def test_row_output_demag_exchange(monkeypatch):
    """The exchange inside the kernel: the rows are of the state, not of Ms times the state."""
    import oracle as O
    n = (2, 12, 20)
    mask = np.random.default_rng(4).uniform(0.5, 1.0, size=n[0] * n[1] * n[2]).astype(np.float32)
    prob = O.full_desc(n=n, cell=(3e-9, 4e-9, 4e-9), demag=1, exchange=0, zeeman=1, msat=8e5, aex=1.3e-11, alpha=0.1,
                       bext=(0.0, 0.01, 0.02), demag_exchange=1, demag_accuracy=2, masks={"msat": mask})
    _compare(monkeypatch, prob, rand_m(n, seed=8), "rk23", 10, masks={"msat": mask}, dt=1e-14, maxerr=1e-5)


@pytest.mark.parametrize("solver", ["rk23", "rk12"])
def test_row_output_time_table(monkeypatch, solver):
    """A field table: the staged scalars of a single plan, at each stage's own time."""
    from mumax2 import Plan
    n = (1, 18, 44)
    prob = dict(n=n, cell=(3e-9, 4e-9, 4e-9), demag=1, exchange=1, zeeman=1, msat=8e5, aex=1.3e-11, alpha=0.1,
                bext=(0.0, 1.0, 1.0), demag_accuracy=2)
    out = []
    for rows in ("0", "1"):
        monkeypatch.setenv("MM_EPI_R2C", rows)
        p = Plan(prob)
        p.solver(solver, dt=1e-13, maxerr=1e-5)
        p.set_state(rand_m(n, seed=6))
        p.set_table("bext", [0.0, 2e-13, 1e-12, 1e-9], [(0, 0, 0), (0, 0.1, 0.3), (0.2, 0.0, 0.1), (0, 0, 0)])
        p.steps(8)
        out.append(p.get_state())
        p.close()
    assert np.array_equal(out[0], out[1])
    assert not np.array_equal(out[0], rand_m(n, seed=6).astype(np.float32))
