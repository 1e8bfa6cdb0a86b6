"""The Q side's EM sums over a long slice (a streamed block's SNPs are one slice): 16,384 positive terms near 2 per individual,
against the formula in 80-bit arithmetic.

The accumulators are folded every 256 SNPs.  Two products per SNP make 512 roundings in a chain and the folds 64 more, each at
most 2^-53 of the sum so far; taken as independent and uniform their root mean square is below
(sqrt(512 / 3) + sqrt(64 / 3)) 2^-53 = 2.0e-15.  One chain of all terms would have sqrt(32768 / 3) 2^-53 = 1.2e-14, half of it
when the sum grows linearly."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", [1, 2, 5, 9, 16])
def test_em_q_over_one_long_slice(oa, K):
    I, J = 64, 16384
    g, _, _ = oa.make_cohort(oa.CohortSpec("t", I, J, K, seed=K, miss=0.02))
    d = oa.AdmixData(I, J, K, 3, rng=K)
    q, p = d.x[:I].astype(np.longdouble), d.x[I:].astype(np.longdouble)
    by = np.asarray(g.data)
    c = np.stack([(by >> (2 * s)) & 3 for s in range(4)], axis=2).reshape(J, -1)[:, :I].T
    dos, nm = np.array([0, 0, 1, 2])[c], c != 1
    qp = q @ p.T
    z1, z2 = np.where(nm, dos / qp, 0), np.where(nm, (2 - dos) / (1 - qp), 0)
    want = q * (z1 @ p + z2 @ (1 - p)) / (2 * J)
    with oa.CuAdmixData(d, g, stream_block=J) as h:
        h.upload(oa.X, d.x)
        oa.em_q(h)
        got = h.download(oa.X_NEXT)[:I]
    err = (got - want) / want
    assert float(np.sqrt(np.mean(err ** 2))) <= 2.0e-15
