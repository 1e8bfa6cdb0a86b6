"""The batched QPs at every group width (4, 8, 16, 32 lanes a problem) and at ragged last blocks: statuses equal the
oracle's quadratic_program! on the device's own sums, and the projected steps agree to 1e-13 (the
same IEEE sequence up to the oracle compiler's contractions)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# tableau rows N = K + 2 (simplex) and K + 1 (box): both sides of each width
@pytest.mark.parametrize("K", [1, 2, 3, 6, 7, 13, 14, 15, 16])
@pytest.mark.parametrize("flags", [0, 1])
def test_qp_groups_match_the_oracle_on_the_same_sums(oa, orc, K, flags):
    I, J = 67, 301
    g, _, _ = oa.make_cohort(oa.CohortSpec("t", I, J, K, seed=K, alpha=0.2))
    d = oa.AdmixData(I, J, K, 3, rng=K + 5)
    with oa.CuAdmixData(d, g, flags=flags) as h:
        h.upload(oa.X, d.x)
        Hq, zq = h.grad_hess_q(oa.X, oa.X)
        st = oa.update_q(d, g, d_cu=h)
        q, p = np.ascontiguousarray(d.x[:I]), np.ascontiguousarray(d.x[I:])
        want, delta = orc.qp_batch(Hq, zq, q, True, orc.MU_GERSHGORIN if flags & 1 else orc.MU_AS_EXECUTED)
        assert np.array_equal(st, want)
        proj = np.stack([orc.project_q1(r) for r in q + delta])
        assert np.max(np.abs(d.x_next[:I] - proj)) < 1e-13
        Hp, zp = h.grad_hess_p(oa.X_NEXT, oa.X)
        st = oa.update_p(d, g, d_cu=h)
        want, delta = orc.qp_batch(Hp, zp, p, False)
        assert np.array_equal(st, want)
        assert np.max(np.abs(d.x_next[I:] - orc.project_p(p + delta))) < 1e-13
