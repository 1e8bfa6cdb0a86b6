"""The mean-imputed FP64 passes (missing cells count with the SNP's mean dosage) at every K: rare and frequent missing cells,
ragged tiles, and lanes whose cells leave the fast range (qp down to 2^-300), observed and imputed ones alike.

Reference: the formulas in numpy.  Each term has at most K + 8 <= 24 roundings, a sum at most 131 terms, on both sides:
2 (24 + 131) 2^-53 = 3.5e-14 of the sum of the terms' magnitudes; asserted at 1e-13."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-13


def _cohort(K, I, J, miss, tiny):
    rng = np.random.default_rng(1000 * K + I)
    q = rng.dirichlet(np.ones(K), I)
    p = rng.uniform(0.1, 0.9, (J, K))
    if tiny:
        one = rng.random(I) < 0.5
        q[one] = np.eye(K)[rng.integers(0, K, one.sum())]
        p[rng.random((J, K)) < 0.2] = 2.0 ** -300
    dos = rng.integers(0, 3, (I, J))
    nm = rng.random((I, J)) >= miss
    nm[0] = True                                      # every SNP has a genotype, so a mean
    code = np.full((-(-I // 4) * 4, J), 1, np.uint8)
    code[:I] = np.where(nm, np.array([0, 2, 3])[dos], 1)
    bed = np.ascontiguousarray((code[0::4] | (code[1::4] << 2) | (code[2::4] << 4) | (code[3::4] << 6)).T)
    mu = (dos * nm).sum(0) / nm.sum(0)
    return q, p, q @ p.T, np.where(nm, dos, mu[None, :]), bed


@pytest.mark.parametrize("K", range(1, 17))
@pytest.mark.parametrize("I,J,miss", [(70, 90, 0.01), (131, 45, 0.4)])
def test_imputed_sums(oa, K, I, J, miss):
    q, p, qp, g, bed = _cohort(K, I, J, miss, False)
    z1, z2 = g / qp, (2 - g) / (1 - qp)
    w1, w2 = z1 / qp, z2 / (1 - qp)
    Hq = np.einsum("ij,jk,jl->ikl", w1, p, p) + np.einsum("ij,jk,jl->ikl", w2, 1 - p, 1 - p)
    Hp = np.einsum("ij,ik,il->jkl", w1 + w2, q, q)
    zq, zp, sp = z1 @ p + z2 @ (1 - p), (z1 - z2).T @ q, (z1 + z2).T @ q
    ll = float((g * np.log(qp) + (2 - g) * np.log(1 - qp)).sum())
    with oa.CuAdmixData(oa.AdmixData(I, J, K, 3, skipmissing=False), oa.Genotypes(bed, I, J)) as h:
        h.upload(oa.X, np.concatenate([q, p]))
        a, b = h.grad_hess_q()
        assert (np.abs(a - Hq) <= TOL * Hq).all() and (np.abs(b - zq) <= TOL * zq).all()
        a, b = h.grad_hess_p(oa.X, oa.X)
        assert (np.abs(a - Hp) <= TOL * Hp).all() and (np.abs(b - zp) <= TOL * sp).all()
        oa.em_q(h)
        oa.em_p(h)
        x = h.download(oa.X_NEXT)
        assert (np.abs(x[:I] - q * zq / (2 * J)) <= TOL * q * zq / (2 * J)).all()
        A, B = p * (z1.T @ q), (1 - p) * (z2.T @ q)
        assert (np.abs(x[I:] - A / (A + B)) <= 4 * TOL).all()
        assert abs(h.loglik() - ll) <= TOL * abs(ll)


@pytest.mark.parametrize("K", range(1, 17))
@pytest.mark.parametrize("I,J,miss", [(70, 90, 0.01), (131, 45, 0.4)])
def test_imputed_loglik_with_lanes_on_both_paths(oa, K, I, J, miss):
    q, p, qp, g, bed = _cohort(K, I, J, miss, True)
    assert (qp < 2.0 ** -255).any()
    ll = float((g * np.log(qp) + (2 - g) * np.log(1 - qp)).sum())
    z1, z2 = g / qp, (2 - g) / (1 - qp)
    zq = z1 @ p + z2 @ (1 - p)
    with oa.CuAdmixData(oa.AdmixData(I, J, K, 3, skipmissing=False), oa.Genotypes(bed, I, J)) as h:
        h.upload(oa.X, np.concatenate([q, p]))
        assert abs(h.loglik() - ll) <= TOL * abs(ll)
        assert (np.abs(h.grad_hess_q()[1] - zq) <= TOL * zq).all()
