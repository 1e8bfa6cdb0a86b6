"""The FP64 sweeps and log-likelihood at the edges of their tiles: 128 rows a CTA, 16 a warp, chunks of 32
columns (16 above K = 8), 8-column pair tiles and 4-cluster products.  Reference: the oracle, at the
1e-10 that the parity tests use, and for points
where qp is exactly 0 or 1 the same formulas in numpy."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FP64_TOL = 1e-10


def _row_rel(a, b):
    """max |a-b| against the row's largest entry; a NaN (0 / 0 in a row without any genotype) has to be in both"""
    a = a.reshape(a.shape[0], -1); b = b.reshape(b.shape[0], -1)
    assert np.array_equal(np.isnan(a), np.isnan(b))
    a, b = np.nan_to_num(a, nan=0.0), np.nan_to_num(b, nan=0.0)
    return float(np.max(np.abs(a - b) / np.maximum(np.abs(b).max(axis=1, keepdims=True), 1e-300)))


# (K, I, J): K at the steps of the pair tiles (T = 1, 6, 10, 15, 36, 45, 78, 91, 136) and of the 4-cluster products
CASES = [(1, 1, 1), (3, 15, 31), (4, 16, 32), (5, 17, 33), (8, 127, 65), (8, 129, 127), (9, 128, 17), (12, 130, 129),
         (13, 33, 500), (16, 257, 63), (2, 700, 1), (16, 1, 300)]


@pytest.mark.parametrize("K,I,J", CASES)
@pytest.mark.parametrize("impute", [False, True])
def test_sums_at_tile_edges_match_oracle(oa, orc, K, I, J, impute):
    g, _, _ = oa.make_cohort(oa.CohortSpec("t", I, J, K, seed=K + I, miss=0.05))
    if impute:   # a SNP without any genotype has no mean
        codes = g.data.copy(); codes[:, 0] = (codes[:, 0] & 0xFC) | 0x02
        g = oa.Genotypes(codes, I, J)
    d = oa.AdmixData(I, J, K, 3, skipmissing=not impute, rng=J)
    q, p = np.ascontiguousarray(d.x[:I]), np.ascontiguousarray(d.x[I:])
    mu = orc.snp_means(g.data, I, J) if impute else None
    with oa.CuAdmixData(d, g) as h:
        h.upload(oa.X, d.x)
        for got, want in ((h.grad_hess_q(), orc.grad_hess_q(g.data, I, J, K, q, p, mu)),
                          (h.grad_hess_p(oa.X, oa.X), orc.grad_hess_p(g.data, I, J, K, q, p, mu))):
            assert _row_rel(got[0], want[0]) < FP64_TOL and _row_rel(got[1], want[1]) < FP64_TOL
        oa.em_q(h); oa.em_p(h)
        x = h.download(oa.X_NEXT)
        assert _row_rel(x[:I], orc.em_q(g.data, I, J, K, q, p, mu)) < FP64_TOL
        assert _row_rel(x[I:], orc.em_p(g.data, I, J, K, q, p, mu)) < FP64_TOL
        ll = orc.loglik(g.data, I, J, K, q, p, mu)
        assert abs(h.loglik() - ll) < FP64_TOL * abs(ll)


@pytest.mark.parametrize("K", [3, 9])
def test_qp_at_zero_and_one(oa, K):
    """Individuals of one cluster and SNPs fixed in it: qp is exactly 0 or 1, where the sums take the division form and
    the log-likelihood a log per cell.  Genotypes agree with the fixed SNPs, so gradients and log-likelihood are
    finite; the Hessians of rows that meet such a cell are NaN."""
    I, J = 70, 90
    rng = np.random.default_rng(K)
    cl = rng.integers(0, K, I)
    q = np.eye(K)[cl]
    p = rng.uniform(0.1, 0.9, (J, K))
    p[rng.random((J, K)) < 0.2] = 0.0
    p[rng.random((J, K)) < 0.2] = 1.0
    qp = p[:, cl].T                                   # exact: one term
    dos = np.where(qp == 0, 0, np.where(qp == 1, 2, rng.integers(0, 3, (I, J))))
    nm = rng.random((I, J)) >= 0.05
    code = np.where(nm, np.array([0, 2, 3])[dos], 1).astype(np.uint8)
    pad = np.full((-(-I // 4) * 4, J), 1, np.uint8); pad[:I] = code
    bed = np.ascontiguousarray((pad[0::4] | (pad[1::4] << 2) | (pad[2::4] << 4) | (pad[3::4] << 6)).T)
    g = oa.Genotypes(bed, I, J)
    with np.errstate(divide="ignore", invalid="ignore"):
        z1 = np.where(nm & (dos > 0), dos / qp, 0.0)
        z2 = np.where(nm & (dos < 2), (2 - dos) / (1 - qp), 0.0)
        w1, w2 = z1 * (1 / qp), z2 * (1 / (1 - qp))   # 0 / 0, as the reference's loops have it: no Hessian there
        ll = float(np.where(nm, np.log(qp ** dos * (1 - qp) ** (2 - dos)), 0.0).sum())
    pp, oo = np.einsum("jk,jl->jkl", p, p), np.einsum("jk,jl->jkl", 1 - p, 1 - p)
    Hq, zq = np.einsum("ij,jkl->ikl", w1, pp) + np.einsum("ij,jkl->ikl", w2, oo), z1 @ p + z2 @ (1 - p)
    Hp, zp = np.einsum("ij,ik,il->jkl", w1 + w2, q, q), (z1 - z2).T @ q
    d = oa.AdmixData(I, J, K, 3)
    with oa.CuAdmixData(d, g) as h:
        h.upload(oa.X, np.concatenate([q, p]))
        a, b = h.grad_hess_q()
        assert _row_rel(a, Hq) < FP64_TOL and _row_rel(b, zq) < FP64_TOL
        a, b = h.grad_hess_p(oa.X, oa.X)
        assert _row_rel(a, Hp) < FP64_TOL
        assert np.max(np.abs(b - zp)) < FP64_TOL * np.abs(zp).max()
        assert abs(h.loglik() - ll) < FP64_TOL * abs(ll)


def test_loglik_is_minus_infinity_where_a_cell_is_impossible(oa):
    I, J, K = 40, 50, 2
    q = np.full((I, K), 0.5); p = np.full((J, K), 0.5); p[7] = 0.0
    bed = np.full((J, 10), 0xAA, np.uint8)            # all heterozygous, at SNP 7 too: qp (1 - qp) = 0
    with oa.CuAdmixData(oa.AdmixData(I, J, K, 3), oa.Genotypes(bed, I, J)) as h:
        h.upload(oa.X, np.concatenate([q, p]))
        assert h.loglik() == -np.inf


@pytest.mark.parametrize("I", [1, 33, 1021, 1024])
def test_caller_owned_columns_any_pitch_and_tail(oa, orc, I):
    """admix_loglik_dev reads columns ceil(I/4) bytes apart, whatever the bits after individual I are."""
    import torch
    from openadmixture_b200 import _native as N
    J, K = 137, 5
    g, _, _ = oa.make_cohort(oa.CohortSpec("t", I, J, K, seed=I))
    want = orc.loglik(g.data, I, J, K, *(lambda x: (np.ascontiguousarray(x[:I]), np.ascontiguousarray(x[I:])))(oa.init_x(I, J, K, 2)))
    data = g.data.copy()
    if I % 4:
        data[:, -1] |= (0xFF << (2 * (I % 4))) & 0xFF
    x = torch.from_numpy(oa.init_x(I, J, K, 2)).cuda()
    bed, out = torch.from_numpy(data).cuda(), torch.zeros(1, dtype=torch.float64, device="cuda")
    n = N.admix_lib().admix_loglik_dev_workspace(I, J, K)
    work = torch.empty(n, dtype=torch.uint8, device="cuda")
    ptr = lambda t: C.c_void_p(t.data_ptr())
    q, p = x[:I].contiguous(), x[I:].contiguous()
    rc = N.admix_lib().admix_loglik_dev(ptr(bed), I, J, K, ptr(q), ptr(p), ptr(out), ptr(work), n,
                                        C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0
    assert abs(out.item() - want) < FP64_TOL * abs(want)
