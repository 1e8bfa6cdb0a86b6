"""The FP64 passes where the lanes of one warp take different paths: a cell whose qp (in the log-likelihood: whose factor) is
below 2^-255 sends its lane's cells through the divisions or the log per cell while the other lanes keep the fast form, and all of
them meet again in the next product.  Every K, the handle's columns and the caller's own.

Reference: the formulas in numpy.  Each term has at most K + 6 <= 22 roundings and a sum at most 90 terms, on both sides
of the comparison: 2 (22 + 90) 2^-53 = 2.5e-14 of the sum of the terms' magnitudes.  Asserted at 1e-13."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-13


def _cohort(K, carried):
    """Individuals of one cluster among mixed ones, and SNPs that are all but absent from a cluster (2^-300); carried: by some
    who have only that cluster, too."""
    I, J = 70, 90
    rng = np.random.default_rng(100 + K)
    q = rng.dirichlet(np.ones(K), I)
    one = rng.random(I) < 0.5
    q[one] = np.eye(K)[rng.integers(0, K, one.sum())]
    p = rng.uniform(0.1, 0.9, (J, K))
    p[rng.random((J, K)) < 0.2] = 2.0 ** -300
    qp = q @ p.T
    dos = np.where((qp < 2.0 ** -255) & (not carried), 0, rng.integers(0, 3, (I, J)))
    nm = rng.random((I, J)) >= 0.05
    code = np.where(nm, np.array([0, 2, 3])[dos], 1).astype(np.uint8)
    pad = np.full((-(-I // 4) * 4, J), 1, np.uint8)
    pad[:I] = code
    bed = np.ascontiguousarray((pad[0::4] | (pad[1::4] << 2) | (pad[2::4] << 4) | (pad[3::4] << 6)).T)
    return I, J, q, p, qp, dos, nm, bed


@pytest.mark.parametrize("K", range(1, 17))
def test_sums_with_lanes_on_both_paths(oa, K):
    I, J, q, p, qp, dos, nm, bed = _cohort(K, False)
    assert 0.02 < (qp < 2.0 ** -255).mean() < 0.5
    z1, z2 = np.where(nm, dos / qp, 0.0), np.where(nm, (2 - dos) / (1 - qp), 0.0)
    w1, w2 = z1 / qp, z2 / (1 - qp)
    pp, oo = np.einsum("jk,jl->jkl", p, p), np.einsum("jk,jl->jkl", 1 - p, 1 - p)
    Hq, zq = np.einsum("ij,jkl->ikl", w1, pp) + np.einsum("ij,jkl->ikl", w2, oo), z1 @ p + z2 @ (1 - p)
    Hp, zp, sp = np.einsum("ij,ik,il->jkl", w1 + w2, q, q), (z1 - z2).T @ q, (z1 + z2).T @ q
    with oa.CuAdmixData(oa.AdmixData(I, J, K, 3), oa.Genotypes(bed, I, J)) as h:
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


@pytest.mark.parametrize("K", range(1, 17))
def test_loglik_with_lanes_on_both_paths(oa, K):
    import torch
    from openadmixture_b200 import _native as N
    I, J, q, p, qp, dos, nm, bed = _cohort(K, True)
    want = float(np.where(nm, dos * np.log(qp) + (2 - dos) * np.log(1 - qp), 0.0).sum())
    with oa.CuAdmixData(oa.AdmixData(I, J, K, 3), oa.Genotypes(bed, I, J)) as h:
        h.upload(oa.X, np.concatenate([q, p]))
        assert abs(h.loglik() - want) <= TOL * abs(want)
    lib, ptr = N.admix_lib(), lambda t: C.c_void_p(t.data_ptr())
    d_bed, d_q, d_p = (torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (bed, q, p))
    out = torch.zeros(2, dtype=torch.float64, device="cuda")
    n = lib.admix_loglik_dev_workspace(I, J, K)
    work = torch.empty(n, dtype=torch.uint8, device="cuda")
    st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert lib.admix_loglik_dev(ptr(d_bed), I, J, K, ptr(d_q), ptr(d_p), ptr(out), ptr(work), n, st) == 0
    assert lib.admix_loglik_dev_noalloc(ptr(d_bed), I, J, K, ptr(d_q), ptr(d_p), ptr(out[1:]), st) == 0
    for got in out.cpu().numpy():
        assert abs(got - want) <= TOL * abs(want)
