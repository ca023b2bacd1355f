"""The convolution passes at the sizes where their stages and tiles change: every length of
the register z multiply, the in-place column transforms at one, two and three stages, prime,
composite and power-of-two lengths, padded and periodic, and the row passes whose lengths are
not powers of two; demag field and torque against the FP64 oracle."""
import pytest

from helpers import rand_m, rel_err, to_np

pytestmark = pytest.mark.gpu

Z_LENGTHS = [(n0, 4, 6) for n0 in range(2, 18)]       # 2..16 in registers, 17 in columns
COLUMNS = [(1, n1, 4) for n1 in (64, 65, 66, 75, 81, 96, 104, 128, 150, 169, 192, 217, 256, 300)]
COLUMNS_3D = [(2, n1, 4) for n1 in (15, 17, 39, 48, 75, 121, 160, 200)] + [(32, 4, 4), (64, 3, 4), (36, 4, 4)]
ROWS = [(1, 4, n2) for n2 in (3, 5, 7, 13, 15, 31, 75, 121, 150, 192, 250, 300, 341)] + [(2, 90, 12), (3, 25, 50)]


# FP32 transforms of L points accumulate about eps * log2(L) <= 12 * 6e-8 relative to the
# largest field: 1e-6 bounds them, with the kernel's own rounding
@pytest.mark.parametrize("n", Z_LENGTHS + COLUMNS + COLUMNS_3D + ROWS)
def test_demag_and_torque_at_size(n):
    import oracle as O
    from mumax2 import Plan
    prob = O.full_desc(n=n, cell=(3e-9, 4e-9, 5e-9), demag=1, exchange=1, msat=8e5, aex=1.3e-11, alpha=0.05,
                       demag_accuracy=2)
    o, g = O.Oracle(prob), Plan(prob)
    m = rand_m(n, seed=sum(n))
    assert rel_err(to_np(g.fields(m)["demag"]), o.fields(m)["demag"]) < 1e-6
    assert rel_err(to_np(g.torque(m)[0]), o.torque(m)[0]) < 2e-6
    g.close()


@pytest.mark.parametrize("n,pbc", [((1, 96, 12), (0, 2, 0)), ((6, 10, 24), (1, 1, 0)), ((12, 6, 20), (2, 0, 1)),
                                   ((1, 256, 8), (0, 1, 1))])
def test_periodic_at_size(n, pbc):
    import oracle as O
    from mumax2 import Plan
    prob = O.full_desc(n=n, cell=(3e-9, 4e-9, 5e-9), pbc=pbc, demag=1, msat=8e5, aex=1.3e-11, demag_accuracy=2)
    o, g = O.Oracle(prob), Plan(prob)
    m = rand_m(n, seed=5)
    assert rel_err(to_np(g.fields(m)["demag"]), o.fields(m)["demag"]) < 1e-6
    g.close()
