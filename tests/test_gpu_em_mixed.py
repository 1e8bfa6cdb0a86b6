"""The Float32 form's EM P-step on small cohorts, at the edges of its tiles of 128 SNPs and chunks of 32 individuals
(tiles of 256 SNPs need more of both).  Reference: the oracle's em_p.

Tolerance on p in [0, 1]: qp and 1 - qp carry 2^-21 relative from the split TF32 products (all terms are positive) and the
tensor core's FP32 accumulation, the reciprocal 2^-22, five FP32 products and an FP32 sum of 16 terms 21 * 2^-24: below
3e-6 per sum.  p' = A / (A + B) moves by at most a quarter of both sums' errors: 2e-6."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

P_TOL = 2e-6

# (K, I, J): one SNP, one individual, either side of 128 and 256 SNPs and of one, two and three chunks
CASES = [(1, 31, 1), (2, 1, 257), (3, 32, 128), (5, 33, 129), (6, 64, 255), (7, 65, 256), (7, 300, 385), (8, 96, 257),
         (8, 97, 130), (9, 129, 127), (12, 161, 129), (16, 95, 300)]


@pytest.mark.parametrize("K,I,J", CASES)
def test_em_p_step_at_tile_edges(oa, orc, K, I, J):
    g, _, _ = oa.make_cohort(oa.CohortSpec("t", I, J, K, seed=K + J, miss=0.04))
    codes = g.data.copy(); codes[:, 0] = (codes[:, 0] & 0xFC) | 0x02      # no SNP without any genotype (0 / 0)
    g = oa.Genotypes(codes, I, J)
    d = oa.AdmixData(I, J, K, 3, rng=I)
    q, p = np.ascontiguousarray(d.x[:I]), np.ascontiguousarray(d.x[I:])
    want = orc.em_p(g.data, I, J, K, q, p)
    with oa.CuAdmixData(d, g, flags=oa.ADMIX_FLAG_MIXED) as h:
        h.upload(oa.X, d.x)
        oa.init_em(d, g, 1, d_cu=h, g_cu=h, quiet=True)
        got = h.download(oa.X)[I:]
    assert np.isfinite(got).all()
    assert np.max(np.abs(got - want)) < P_TOL
