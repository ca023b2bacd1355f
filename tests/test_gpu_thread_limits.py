"""Two host threads that drive plans, or weight gradients, of different sizes through the same
kernels: the launches of one must not lower the shared-memory limit that the other's need."""
import ctypes as C
import threading

import pytest

from helpers import rand_m, rel_err, to_np

pytestmark = pytest.mark.gpu


def _both(jobs):
    """Runs the jobs in one thread each; the errors that they raised."""
    errors = []
    start = threading.Barrier(len(jobs))

    def work(job):
        try:
            start.wait()
            job()
        except Exception as e:  # handed to the caller
            errors.append(str(e))

    ts = [threading.Thread(target=work, args=(j,)) for j in jobs]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    return errors


# columns (600 and 1500 rows), rows (1500 and 2000 cells), row tiles of one power-of-two length
@pytest.mark.parametrize("sizes", [((1, 600, 8), (1, 1500, 8)), ((1, 4, 1500), (1, 4, 2000)),
                                   ((2, 600, 8), (2, 1500, 8)), ((1, 150, 1024), (1, 750, 1024))])
def test_plans_of_two_sizes(sizes):
    import torch
    from mumax2 import Plan
    from mumax2 import _native as nat
    p = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    plans, states, alone, out = [], [], [], []
    for n in sizes:
        prob = dict(n=n, cell=(3e-9, 4e-9, 4e-9), demag=1, exchange=1, msat=8e5, aex=1.3e-11, alpha=0.1,
                    demag_accuracy=1)
        plans.append(Plan(prob))
        t, m = plans[-1].torque(rand_m(n, seed=sum(n)))
        states.append(m)
        alone.append(plans[-1].torque(m)[0])
        out.append(torch.zeros_like(t))

    def job(k):
        for _ in range(1000):
            nat.check(nat.lib().mm_torque(plans[k].h, p(states[k]), 0, 0.0, p(out[k]), None))

    assert not _both([lambda: job(0), lambda: job(1)])
    torch.cuda.synchronize()
    for k in range(2):
        # every call normalises the state again: a few roundings of 6e-8
        assert rel_err(to_np(out[k]), to_np(alone[k])) < 1e-5
        plans[k].close()


def test_weight_gradients_of_two_widths():
    import torch
    from mumax2 import _native as nat
    p = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    cin, cout = 32, 32
    data, out = [], []
    for B, H, W in ((64, 64, 64), (4, 128, 400)):
        x = torch.randn(B * H * W, cin, device="cuda").bfloat16()
        dy = torch.randn(B * H * W, cout, device="cuda").bfloat16()
        data.append((x, dy, B, H, W))
        out.append(torch.zeros(cout * 9 * cin, device="cuda"))

    def job(k):
        x, dy, B, H, W = data[k]
        for _ in range(1000):
            nat.check(nat.lib().mm_nn_conv3x3_wgrad(p(dy), cout, 0, cout, p(x), cin, 0, cin, p(out[k]), B, H, W, None))

    assert not _both([lambda: job(0), lambda: job(1)])
    torch.cuda.synchronize()
