"""The sketch at the edges of its kernel: blocks of 4 individuals (one byte of the columns), a thread every 256th sketch
SNP with the next SNP's byte and the one after's index in flight, so the branches turn at 256 and 512 SNPs.  Reference: the
oracle.  Dosages and frequencies (ratios of exact integers, rounded once) are equal; a projection is an FP32 sum of S terms, each
sum and term within 2^-22 S of the largest, as in the other sketch test."""
import sys
from pathlib import Path

import numpy as np
import pytest

sys.path.insert(0, str(Path(__file__).resolve().parent.parent / "oracle"))
import mlp_oracle as mo  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S", [1, 2, 255, 256, 257, 511, 512, 513, 769])
@pytest.mark.parametrize("I", [1, 2, 3, 4, 5, 9])
def test_sketch_strides(oa, I, S):
    from openadmixture_b200 import warmstart as ws
    J, R = S + 5, 32
    g = oa.Genotypes(np.random.default_rng(S).integers(0, 256, (J, (I + 3) // 4)).astype(np.uint8), I, J)
    snps = np.sort(np.random.default_rng(I).choice(J, S, replace=False)).astype(np.int32)
    sk = ws.sketch(g, snps, R=R, seed=5)
    freq, dos, proj = mo.sketch(g.data, I, snps, R, 5)
    assert np.array_equal(sk.dos.cpu().numpy(), dos)
    assert np.array_equal(sk.freq.cpu().numpy(), freq)
    z = np.abs(proj).max(initial=0.0) + 1.0
    assert np.abs(sk.proj.cpu().numpy() - proj).max(initial=0.0) <= 2.0 ** -22 * S * z
