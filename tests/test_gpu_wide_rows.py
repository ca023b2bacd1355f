"""Rows of 2048 cells, which transform at 4096 points: field, torque and time steps against the FP64
oracle."""
import numpy as np
import pytest

from helpers import rand_m, rel_err, to_np

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(1, 4, 2048), (2, 3, 2048)])
def test_field_torque_and_steps(n):
    import oracle as O
    from mumax2 import Plan
    prob = O.full_desc(n=n, cell=(3e-9, 4e-9, 5e-9), demag=1, exchange=1, zeeman=1, bext=(0.0, 0.01, 0.02), msat=8e5,
                       aex=1.3e-11, alpha=0.05, demag_accuracy=2)
    o, g = O.Oracle(prob), Plan(prob)
    m = rand_m(n, seed=sum(n))
    # the bounds of test_gpu_sizes: FP32 transforms of up to 4096 points, eps * log2(L) each way
    assert rel_err(to_np(g.fields(m)["demag"]), o.fields(m)["demag"]) < 1e-6
    assert rel_err(to_np(g.torque(m)[0]), o.torque(m)[0]) < 2e-6
    r = O.OracleRun(o, m, solver="rk23", dt=1e-14, maxerr=1e-5)
    g.solver("rk23", dt=1e-14, maxerr=1e-5)
    g.set_state(m)
    for _ in range(3):
        r.step()
    g.steps(3)
    assert np.abs(to_np(g.get_state()) - r.m).max() < 2e-5   # the trajectory bar of a few steps
    g.close()
