"""A NaN in a hidden layer reaches the probabilities and the loss: the ReLU keeps it (max(NaN, 0) would be 0), as the
oracle's numpy maximum does.  This is how a product whose bounded wait ran out shows.  One, two and eight CTAs per tile."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [40, 2048, 10240])
@pytest.mark.parametrize("name", ["w1", "w2", "b1"])
def test_nan_reaches_the_loss(oa, n, name):
    import torch
    from openadmixture_b200 import warmstart as W
    S, R, K = 1000, 32, 8
    rng = np.random.default_rng(n)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    sk = W.Sketch(t(rng.integers(0, 3, (n, S)).astype(np.int8)), t(rng.uniform(0.05, 0.95, S).astype(np.float32)),
                  t(rng.normal(size=(n, R)).astype(np.float32)))
    m = W.WarmStartMLP(S, R, K, 256, seed=2, snps=np.arange(S))
    assert torch.isfinite(m.forward(sk)).all()
    m.p[name].view(-1)[5] = float("nan")
    assert torch.isnan(m.forward(sk)).all()
    loss = W.train(m, [(sk, t(rng.dirichlet(np.ones(K), n).astype(np.float32)))], epochs=1, batch=n)
    assert np.isnan(loss[0])
