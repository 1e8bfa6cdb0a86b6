"""The FP64 sweeps' reciprocal of qp and of 1 - qp against 1.0 / x.  With one cluster, Q = 1 and one genotype per SNP the P-side
gradient is 2 / qp (dosage 2) or -2 / (1 - qp) (dosage 0) and nothing else, so it shows the reciprocal itself.

In [2^-255, 2) it is the hardware's estimate r, good to 20 bits, and one third-order step r (1 + e + e^2), e = 1 - x r: what
is left is e^3 = 2^-60, 2^-7 of an ulp, before the last rounding.  So it is at most one ulp from the correctly rounded
quotient; below that range the quotient is IEEE division, equal to numpy's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _gradients(oa, p, code):
    """sum_i z1 - z2 of every SNP: individual 0 has the code, 31 others are missing"""
    I, J = 32, len(p)
    bed = np.full((J, 8), 0x55, np.uint8)
    bed[:, 0] = 0x54 | code
    with oa.CuAdmixData(oa.AdmixData(I, J, 1, 3), oa.Genotypes(bed, I, J)) as h:
        h.upload(oa.X, np.concatenate([np.ones((I, 1)), p[:, None]]))
        return h.grad_hess_p(oa.X, oa.X)[1][:, 0]


def _ulps(got, x):
    want = 1.0 / x
    return np.abs(got - want) / np.spacing(want)


def _values():
    rng = np.random.default_rng(1)
    two = 2.0 ** -np.arange(1.0, 256.0)
    near = np.concatenate([two * (1 + k * 2.0 ** -52) for k in (0, 1, 2, 3)] + [two[:-1] * (1 - k * 2.0 ** -53) for k in (1, 2, 3)])
    return np.concatenate([near, 1e-5 * (1 + rng.uniform(-1e-3, 1e-3, 2000)), [1 - 2.0 ** -53, 1 - 2.0 ** -52, 2.0 ** -255],
                           rng.uniform(1e-5, 1, 60000), 2.0 ** rng.uniform(-255, 0, 20000)])


def test_reciprocal_of_qp(oa):
    p = _values()
    assert p.min() == 2.0 ** -255 and p.max() < 1.0
    assert _ulps(_gradients(oa, p, 3) / 2, p).max() <= 1.0


def test_reciprocal_of_one_minus_qp(oa):
    x = _values()
    p = np.concatenate([x, 1 - x[x >= 2.0 ** -53], 1 - 2.0 ** -np.arange(1.0, 54.0)])
    p = p[p < 1.0]
    assert _ulps(_gradients(oa, p, 0) / -2, 1 - p).max() <= 1.0


def test_below_the_range_it_divides(oa):
    rng = np.random.default_rng(2)
    p = np.concatenate([2.0 ** -255 * (1 - 2.0 ** -53 * np.array([1.0, 2.0, 3.0])), 2.0 ** rng.uniform(-1000, -255.001, 5000)])
    assert np.array_equal(_gradients(oa, p, 3) / 2, 1.0 / p)
