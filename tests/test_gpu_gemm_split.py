"""The encoder's products where one output tile is shared by 8 or 2 CTAs (few tiles, a long reduction): either side of
24 and 74 tiles and of the reduction's block counts.

Forward: every individual's row is a product of its own, and a split adds the same blocks in the same order, so a
small batch's probabilities equal, bit for bit, those of the same individuals in a batch too large to split.
Backward: the last layer's weight gradient against FP64 products of the device's own operands.  Its products carry 2^-17
(two BF16 parts each), its sums at most 24 truncating accumulations per block and one FP32 addition per block (58 in
all, each 2^-23): 2^-16 of sum |h2| |dlogits|."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _model(S):
    from openadmixture_b200 import warmstart as W
    return W, W.WarmStartMLP(S, 32, 8, 256, seed=3, snps=np.arange(S))


@pytest.mark.parametrize("S", [64, 97, 300, 1000, 4096])      # 1, 2, 3, 9 and 33 blocks in the first layer
def test_split_forward_is_bitwise_the_unsplit_one(oa, S):
    torch = pytest.importorskip("torch")
    W, m = _model(S)
    rng = np.random.default_rng(S)
    n = 10240                                                # 320 tiles
    dos = torch.from_numpy(rng.integers(0, 4, (n, S)).astype(np.int8)).cuda()
    proj = torch.from_numpy(rng.normal(size=(n, 32)).astype(np.float32)).cuda()
    freq = torch.from_numpy(rng.uniform(0.05, 0.95, S).astype(np.float32)).cuda()
    full = m.forward(W.Sketch(dos, freq, proj)).cpu().numpy()
    assert np.isfinite(full).all()
    for k in (1, 127, 129, 768, 769, 2304, 2305, 4096):      # 4, 4, 8, 24, 28, 72, 76 and 128 tiles
        part = m.forward(W.Sketch(dos[:k].contiguous(), freq, proj[:k].contiguous())).cpu().numpy()
        assert np.array_equal(part, full[:k]), k


@pytest.mark.parametrize("n", [129, 1000, 4096, 4225, 9001])  # 2, 8, 32, 34 (rounds of 24 and 10) and 71 blocks
def test_split_weight_gradient_matches_fp64(oa, n):
    torch = pytest.importorskip("torch")
    from openadmixture_b200 import _native as N
    W, m = _model(200)
    rng = np.random.default_rng(n)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    e = lambda *s: torch.empty(s, dtype=torch.float32, device="cuda")
    p = lambda x: C.c_void_p(x.data_ptr())
    dos, proj = t(rng.integers(0, 4, (n, 200)).astype(np.int8)), t(rng.normal(size=(n, 32)).astype(np.float32))
    cen, tgt = t(rng.random(200).astype(np.float32)), t(rng.dirichlet(np.ones(8), n).astype(np.float32))
    h1, h2, d1, d2, lg, pr, dl, loss = e(n, 256), e(n, 256), e(n, 256), e(n, 256), e(n, 8), e(n, 8), e(n, 8), e(1)
    g = {k: torch.zeros_like(v) for k, v in m.p.items()}
    G = N.MLPGrads(*[g[k].data_ptr() for k in W.WarmStartMLP.NAMES])
    net, lib, st = m.net(), N.admix_lib(), C.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert lib.admix_mlp_forward(C.byref(net), n, p(dos), p(cen), p(proj), p(h1), p(h2), p(lg), p(pr), st) == 0
    assert lib.admix_mlp_backward(C.byref(net), C.byref(G), n, p(dos), p(cen), p(proj), p(h1), p(h2), p(lg), p(tgt),
                                  p(pr), p(dl), p(d2), p(d1), p(loss), st) == 0
    torch.cuda.synchronize()
    a, b = h2.double(), dl.double()
    err = (g["w3"].double() - a.T @ b).abs()
    assert bool((err <= 2.0 ** -16 * (a.abs().T @ b.abs()) + 1e-30).all())
