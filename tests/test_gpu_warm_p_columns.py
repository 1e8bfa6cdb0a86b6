"""The learned start's P step on the caller's own columns at any base alignment and with few columns, where the first and the
last column's blocks are read bytewise.  Bit for bit the serial FP32 sums: a dosage 0, 1 or 2 times q is exact, so every add
rounds once, in the order of the individuals."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("I,J,K", [(64, 1, 2), (65, 2, 3), (130, 6, 8), (257, 127, 1), (321, 130, 5), (1021, 258, 12)])
@pytest.mark.parametrize("off", [0, 1, 2, 3])
def test_any_base_alignment(oa, I, J, K, off):
    import torch
    from openadmixture_b200 import _native as N
    rng = np.random.default_rng(I + off)
    Ib = (I + 3) // 4
    raw = rng.integers(0, 256, off + J * Ib).astype(np.uint8)
    q = rng.dirichlet(np.ones(K), I)
    by = raw[off:].reshape(J, Ib)
    c = np.stack([(by >> (2 * s)) & 3 for s in range(4)], axis=2).reshape(J, -1)[:, :I].T
    dos, nm = np.array([0, 0, 1, 2], np.float32)[c], np.array([1, 0, 1, 1], np.float32)[c]
    q32 = q.astype(np.float32)
    num, den = np.zeros((J, K), np.float32), np.zeros((J, K), np.float32)
    for i in range(I):
        num += dos[i][:, None] * q32[i][None, :]
        den += nm[i][:, None] * q32[i][None, :]
    want = np.clip(num.astype(np.float64) / (2 * den).astype(np.float64), 1e-5, 1 - 1e-5)
    buf, d_q = torch.from_numpy(raw).cuda(), torch.from_numpy(q).cuda()
    p = torch.empty((J, K), dtype=torch.float64, device="cuda")
    st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert N.admix_lib().admix_warm_p(C.c_void_p(buf.data_ptr() + off), Ib, I, J, K, C.c_void_p(d_q.data_ptr()),
                                      C.c_void_p(p.data_ptr()), st) == 0
    assert np.array_equal(p.cpu().numpy(), want)
