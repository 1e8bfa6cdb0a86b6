"""The batched QPs where there are more than the GPU has lanes for: one thread solves a problem there (K up to 4).  A problem's
answer does not depend on how many others there are, so a slice of a large batch equals, bit for bit, the same problems solved
by groups of lanes.  The second axis is one slice of partial sums in both (40 columns)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SMALL, OTHER = 1003, 40


def _data(oa, I, J, K, x):
    d = oa.AdmixData(I, J, K, 3)
    d.x[:] = x
    d.x_next[:] = x
    return d


# problems on either side of the rule: 148 SMs x 2,048 threads over 4 lanes a problem (half as many for K <= 2), 8 lanes
@pytest.mark.parametrize("K,n", [(1, 40000), (2, 38001), (3, 80000), (4, 40001), (4, 37000), (5, 80000)])
@pytest.mark.parametrize("flags", [0, 1])
def test_box_problems(oa, K, n, flags):
    g, _, _ = oa.make_cohort(oa.CohortSpec("t", OTHER, n, K, seed=K, alpha=0.2, miss=0.05))
    x = oa.init_x(OTHER, n, K, K + 3)
    d = _data(oa, OTHER, n, K, x)
    with oa.CuAdmixData(d, g, flags=flags) as h:
        st = oa.update_p(d, g, d_cu=h)
    for a in (0, n - SMALL):
        gs = oa.Genotypes(np.ascontiguousarray(g.data[a:a + SMALL]), OTHER, SMALL)
        ds = _data(oa, OTHER, SMALL, K, np.concatenate([x[:OTHER], x[OTHER + a:OTHER + a + SMALL]]))
        with oa.CuAdmixData(ds, gs, flags=flags) as h:
            sts = oa.update_p(ds, gs, d_cu=h)
        assert np.array_equal(st[a:a + SMALL], sts)
        assert np.array_equal(d.x_next[OTHER + a:OTHER + a + SMALL], ds.x_next[OTHER:])


@pytest.mark.parametrize("K,n", [(1, 40000), (2, 38004), (3, 40000), (4, 40004), (4, 37000), (5, 80000)])
@pytest.mark.parametrize("flags", [0, 1])
def test_simplex_problems(oa, K, n, flags):
    g, _, _ = oa.make_cohort(oa.CohortSpec("t", n, OTHER, K, seed=K, alpha=0.2, miss=0.05))
    x = oa.init_x(n, OTHER, K, K + 3)
    d = _data(oa, n, OTHER, K, x)
    with oa.CuAdmixData(d, g, flags=flags) as h:
        st = oa.update_q(d, g, d_cu=h)
    m = SMALL // 4 * 4
    for a in (0, n - m):                                  # whole bytes of the columns
        gs = oa.Genotypes(np.ascontiguousarray(g.data[:, a // 4:(a + m) // 4]), m, OTHER)
        ds = _data(oa, m, OTHER, K, np.concatenate([x[a:a + m], x[n:]]))
        with oa.CuAdmixData(ds, gs, flags=flags) as h:
            sts = oa.update_q(ds, gs, d_cu=h)
        assert np.array_equal(st[a:a + m], sts)
        assert np.array_equal(d.x_next[a:a + m], ds.x_next[:m])
