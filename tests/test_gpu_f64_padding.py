"""Rows that take the placeholder coefficients of cells past a tile's columns to qp = 1: any Q and P may be uploaded, so a
row of Q that sums to 2 meets them there on the Q side and a SNP whose P averages 2 on the P side.  Those cells are nobody's:
the sums are those of the real cells alone, as a loop over them has it (numpy; at most 70 terms of one sign in the Hessian
and in the Q sums, 2 (70 + 20) 2^-53 = 2e-14, asserted at 1e-13 of the terms' magnitudes)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-13


def _bed(rng, I, J):
    dos, nm = rng.integers(0, 3, (I, J)), rng.random((I, J)) >= 0.1
    code = np.full((-(-I // 4) * 4, J), 1, np.uint8)
    code[:I] = np.where(nm, np.array([0, 2, 3])[dos], 1)
    return np.ascontiguousarray((code[0::4] | (code[1::4] << 2) | (code[2::4] << 4) | (code[3::4] << 6)).T), dos, nm


@pytest.mark.parametrize("K", [1, 2, 4, 8, 9, 16])
@pytest.mark.parametrize("I,J", [(5, 33), (33, 5), (50, 70)])
def test_q_rows_that_sum_to_two(oa, K, I, J):
    rng = np.random.default_rng(K)
    bed, dos, nm = _bed(rng, I, J)
    q = np.full((I, K), 2.0 / K)
    p = rng.integers(1, 16, (J, K)) / 64.0                # qp is exact, in [1/32, 1/2)
    qp = q @ p.T
    z1, z2 = np.where(nm, dos / qp, 0.0), np.where(nm, (2 - dos) / (1 - qp), 0.0)
    w1, w2 = z1 / qp, z2 / (1 - qp)
    H = np.einsum("ij,jk,jl->ikl", w1, p, p) + np.einsum("ij,jk,jl->ikl", w2, 1 - p, 1 - p)
    z = z1 @ p + z2 @ (1 - p)
    with oa.CuAdmixData(oa.AdmixData(I, J, K, 3), oa.Genotypes(bed, I, J)) as h:
        h.upload(oa.X, np.concatenate([q, p]))
        a, b = h.grad_hess_q()
        assert (np.abs(a - H) <= TOL * H).all() and (np.abs(b - z) <= TOL * z).all()


@pytest.mark.parametrize("K", [2, 4, 8, 16])
@pytest.mark.parametrize("I,J", [(5, 33), (33, 5), (50, 70)])
def test_snps_whose_p_averages_two(oa, K, I, J):
    rng = np.random.default_rng(K + 50)
    bed, dos, nm = _bed(rng, I, J)
    q = np.eye(K)[rng.integers(0, K, I)]
    p = np.tile([1.5, 2.5], (J, K // 2))
    qp = q @ p.T
    z1, z2 = np.where(nm, dos / qp, 0.0), np.where(nm, (2 - dos) / (1 - qp), 0.0)
    w = z1 / qp + z2 / (1 - qp)
    H, z, s = np.einsum("ij,ik,il->jkl", w, q, q), (z1 - z2).T @ q, (np.abs(z1) + np.abs(z2)).T @ q
    with oa.CuAdmixData(oa.AdmixData(I, J, K, 3), oa.Genotypes(bed, I, J)) as h:
        h.upload(oa.X, np.concatenate([q, p]))
        a, b = h.grad_hess_p(oa.X, oa.X)
        assert (np.abs(a - H) <= TOL * np.abs(H)).all() and (np.abs(b - z) <= TOL * s).all()
