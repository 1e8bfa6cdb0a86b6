"""The SNP selection spread over a cluster of eight blocks per list, and the device-side standardisation: identical to
the oracle for lists shorter than the blocks, ties across block borders, nearly everything kept, and SNPs
without variance or without genotypes."""
import sys
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

sys.path.insert(0, str(Path(__file__).resolve().parents[1] / "oracle"))
import skfr_oracle as S  # noqa: E402


@pytest.mark.parametrize("J,s", [(5, 2), (31, 31), (32, 1), (4099, 4098), (9001, 700)])
@pytest.mark.parametrize("mode", ["global", "local"])
def test_selection_spread_over_blocks(oa, J, s, mode):
    I, K = 60, 3
    data = oa.make_cohort(oa.CohortSpec("t", I, J, K, seed=J, alpha=0.1))[0].data.copy()
    data[J // 2: 2 * (J // 2)] = data[: J // 2]          # equal scores far apart: ties go to the lower SNP
    data[J // 3] = 0x00                                  # no variance
    data[J // 4] = 0x55                                  # no genotype
    c, aims, obj, it = oa.skfr(oa.Genotypes(data, I, J), K, s, mode=mode, max_iter=4, rng=1)
    c_o, aims_o, obj_o, it_o = S.skfr(data, I, K, s, mode=mode, max_iter=4, seed=1)
    assert np.array_equal(c, c_o) and np.array_equal(aims, aims_o) and it == it_o
    assert obj == pytest.approx(obj_o, rel=1e-12)
