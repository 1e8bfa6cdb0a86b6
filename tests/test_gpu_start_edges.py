"""The learned start's kernels at ragged sizes and alignments: sketches whose blocks of 4 individuals and strides of 256
SNPs do not come out even, columns at any pitch, SNP pairs, 64-individual chunks, and products whose
input rows are not 8-byte aligned."""
import sys
from pathlib import Path

import numpy as np
import pytest

sys.path.insert(0, str(Path(__file__).resolve().parent.parent / "oracle"))
import mlp_oracle as mo  # noqa: E402

pytestmark = pytest.mark.gpu


def _genotypes(oa, I, J, seed):
    """random codes, garbage past individual I in the last byte"""
    return oa.Genotypes(np.random.default_rng(seed).integers(0, 256, (J, (I + 3) // 4)).astype(np.uint8), I, J)


@pytest.mark.parametrize("I,S,R", [(1, 1, 1), (31, 15, 32), (32, 16, 32), (33, 17, 5), (130, 160, 31), (257, 1001, 3), (40, 16400, 32)])
def test_sketch_edges(oa, I, S, R):
    from openadmixture_b200 import warmstart as ws
    g = _genotypes(oa, I, S + 3, I)
    snps = np.sort(np.random.default_rng(1).choice(S + 3, S, replace=False)).astype(np.int32)
    sk = ws.sketch(g, snps, R=R, seed=5)
    freq, dos, proj = mo.sketch(g.data, I, snps, R, 5)
    assert np.array_equal(sk.dos.cpu().numpy(), dos)
    assert np.array_equal(sk.freq.cpu().numpy(), freq)          # a ratio of exact integers, rounded once to FP32
    # FP32 sums of S terms of magnitude at most 1 / sqrt(1e-6) (a frequency at 0 or 1), scaled by S^-1/2
    z = np.abs(proj).max(initial=0.0) + 1.0
    assert np.abs(sk.proj.cpu().numpy() - proj).max(initial=0.0) <= 2.0 ** -22 * S * z


@pytest.mark.parametrize("I,J,K", [(1, 1, 1), (63, 2, 2), (64, 127, 3), (65, 128, 4), (130, 129, 5), (257, 260, 8),
                                   (1000, 5, 15), (1021, 3, 16)])
def test_warm_p_is_the_serial_fp32_sum(oa, I, J, K):
    from openadmixture_b200 import warmstart as ws
    g = _genotypes(oa, I, J, J)
    q = np.random.default_rng(K).dirichlet(np.ones(K), I)
    c = mo.codes(g.data, I)
    dos, nm = np.array([0, 0, 1, 2], np.float32)[c], np.array([1, 0, 1, 1], np.float32)[c]
    q32 = q.astype(np.float32)
    num, den = np.zeros((J, K), np.float32), np.zeros((J, K), np.float32)
    for i in range(I):                                          # dosage 0, 1, 2 times q is exact: one rounding per add
        num += dos[i][:, None] * q32[i][None, :]
        den += nm[i][:, None] * q32[i][None, :]
    with np.errstate(invalid="ignore", divide="ignore"):
        want = np.where(den > 0, num.astype(np.float64) / (2 * den).astype(np.float64), 0.5)
    assert np.array_equal(ws.warm_p(g, q), np.clip(want, 1e-5, 1 - 1e-5))


@pytest.mark.parametrize("n,S,R,H,K", [(1, 7, 1, 8, 2), (127, 8, 0, 65, 3), (129, 31, 32, 64, 5), (300, 130, 5, 33, 16)])
def test_forward_at_ragged_products(oa, n, S, R, H, K):
    import ctypes as C
    import torch
    from openadmixture_b200 import _native as N, warmstart as ws
    rng = np.random.default_rng(S)
    dos = rng.integers(0, 4, (n, S)).astype(np.int8)
    center, proj = rng.uniform(0.1, 1.9, S).astype(np.float32), rng.normal(0, 1, (n, R)).astype(np.float32)
    m = ws.WarmStartMLP(S, R, K, H=H, seed=n)
    *_, want = mo.forward(m.numpy_params(), dos, center.astype(np.float64), proj)
    t = lambda a: torch.tensor(a, device="cuda")  # noqa: E731
    P = lambda x: C.c_void_p(x.data_ptr())  # noqa: E731
    d, c, p = t(dos), t(center), t(np.ascontiguousarray(proj) if R else np.zeros((n, 1), np.float32))
    h1, lg = torch.empty((n, H), device="cuda"), torch.empty((n, K), device="cuda")
    h2, pr = torch.empty_like(h1), torch.empty_like(lg)
    net = m.net()
    assert N.admix_lib().admix_mlp_forward(C.byref(net), n, P(d), P(c), P(p), P(h1), P(h2), P(lg), P(pr), None) == 0
    torch.cuda.synchronize()
    assert np.allclose(pr.cpu().numpy(), want, atol=2e-5)
