"""Rows whose lengths are not powers of two, at every number of lines that a block takes: 1, 2, 4,
8 and 16 rows in the row pass, 3, 6 and 15 lines in the epilogue, with and without a radix above
10; the field against the convolution with the plan's own kernel in FP64, and the epilogue's row
output against the row pass."""
import numpy as np
import pytest

from helpers import rand_m, rel_err, to_np
from test_gpu_epi_r2c import _compare
from test_gpu_long_columns import _field64

pytestmark = pytest.mark.gpu

SIZES = [(1, 5, 12), (1, 5, 22), (1, 600, 12), (1, 600, 13), (1, 1500, 6), (1, 1500, 11), (4, 400, 24), (6, 1000, 10),
         (1, 1500, 75)]


def _prob(n):
    import oracle as O
    return O.full_desc(n=n, cell=(3e-9, 4e-9, 5e-9), demag=1, exchange=1, msat=8e5, aex=1.3e-11, alpha=0.05,
                       demag_accuracy=1)


# the bound of test_gpu_sizes: FP32 transforms of up to 4096 points, eps * log2(L) each way
@pytest.mark.parametrize("n", SIZES)
def test_field(n):
    from mumax2 import Plan
    g = Plan(_prob(n))
    m = rand_m(n, seed=sum(n)).astype(np.float32)
    want = _field64(g, n, (0, 0, 0), m, np.ones(n[0] * n[1] * n[2], np.float32), 8e5)
    assert rel_err(to_np(g.fields(m)["demag"]), want) < 1e-6
    g.close()


@pytest.mark.parametrize("n", SIZES)
def test_row_output(monkeypatch, n):
    _compare(monkeypatch, _prob(n), rand_m(n, seed=3), "rk23", 6, dt=1e-13, maxerr=1e-5)
