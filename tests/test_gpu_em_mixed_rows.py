"""The Float32 form's EM P-step where a CTA owns 256 SNPs (many SNPs and individuals, K up to 8) and where it owns 128: ragged
last tiles and slices, and streamed blocks.  A SNP's step depends on its own column alone, so the oracle is asked for the
first SNPs and for the last tiles only.

Tolerance on p in [0, 1] as for one tile: qp and 1 - qp carry 2^-21 relative, the reciprocal 2^-22, five FP32 products and
an FP32 sum of 16 terms 21 * 2^-24, chunks are added in FP64: below 3e-6 per sum, and p' = A / (A + B) moves by at most a
quarter of both sums' errors: 2e-6."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

P_TOL = 2e-6


def _step(oa, g, d, **kw):
    with oa.CuAdmixData(d, g, flags=oa.ADMIX_FLAG_MIXED, **kw) as h:
        h.upload(oa.X, d.x)
        oa.init_em(d, g, 1, d_cu=h, g_cu=h, quiet=True)
        return h.download(oa.X)[g.I:]


@pytest.mark.parametrize("K,I,J", [(1, 12001, 20001), (3, 11999, 20223), (5, 12031, 20225), (7, 12000, 20353), (8, 12033, 20479),
                                   (5, 400, 20225), (8, 5000, 5001)])
def test_em_p_step_of_many_snps(oa, orc, K, I, J):
    spec = oa.CohortSpec("t", I, J, K, seed=K, miss=0.04)
    q_true, p_true = oa.truth(spec)
    g = oa.genotypes_device(spec, q_true, p_true).to_host()
    d = oa.AdmixData(I, J, K, 3, rng=I)
    q, p = d.x[:I].copy(), d.x[I:].copy()         # the step writes d.x
    got = _step(oa, g, d)
    assert np.isfinite(got).all()
    for s in (slice(0, 40), slice(J - 300, J)):
        want = orc.em_p(np.ascontiguousarray(g.data[s]), I, s.stop - s.start, K, q, np.ascontiguousarray(p[s]))
        assert np.max(np.abs(got[s] - want)) < P_TOL


@pytest.mark.parametrize("block", [1024, 65536])            # 8 tiles of 128, 313 of 256 in the first block
def test_em_p_step_of_streamed_blocks(oa, orc, block):
    K, I, J = 4, 900, 80100
    spec = oa.CohortSpec("t", I, J, K, seed=K, miss=0.04)
    q_true, p_true = oa.truth(spec)
    g = oa.genotypes_device(spec, q_true, p_true).to_host()
    d = oa.AdmixData(I, J, K, 3, rng=I)
    q, p = d.x[:I].copy(), d.x[I:].copy()         # the step writes d.x
    got = _step(oa, g, d, stream_block=block)
    for s in (slice(0, 40), slice(65400, 65700), slice(J - 300, J)):
        want = orc.em_p(np.ascontiguousarray(g.data[s]), I, s.stop - s.start, K, q, np.ascontiguousarray(p[s]))
        assert np.max(np.abs(got[s] - want)) < P_TOL
