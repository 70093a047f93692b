"""The training launch over tiles, steps and launches: ragged last batches, more
tiles than resident blocks, more steps than one launch holds. With a vanishing
step size an epoch's loss is the loss of the whole set (the sums differ in the
order of their doubles only); a first step of one batch moves every parameter by
the step size times g / (|g| + eps) of the whole set's gradient."""
import numpy as np
import pytest

import troute_gb300 as T

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def pairs_of(n, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    q = torch.exp(torch.randn((n, 4), generator=g, device="cuda"))
    u = torch.rand((n, 4), generator=g, device="cuda")
    rest = torch.stack([500 + 4500 * u[:, 0], 1e-5 + 1e-2 * u[:, 1], 0.03 + 0.05 * u[:, 2], 2 + 48 * u[:, 3],
                        0.3 * q[:, 1] ** 0.6 + 0.1], 1)
    return torch.cat([q, rest], 1).float().contiguous()


@pytest.mark.parametrize("n,batch", [(2, 64), (63, 64), (64, 64), (65, 64), (1000, 320), (20001, 6400), (40000, 20480),
                                     (4_300_000, 64)])
def test_epoch_loss_is_the_loss_of_all_pairs(n, batch):
    p = pairs_of(n, n)
    m = T.WarmModel(3)
    loss = m.fit(p.data_ptr(), n, epochs=2, batch=batch, lr=1e-30, weight_decay=0.0, seed=5)
    want = m.grad(p.cpu().numpy())[1]
    assert np.all(np.abs(loss - want) <= 1e-6 * want)


@pytest.mark.parametrize("n,batch", [(2, 64), (65, 128), (9729, 9792), (20001, 20480)])
def test_first_step(n, batch):
    p = pairs_of(n, n + 1)
    a, b = T.WarmModel(4), T.WarmModel(4)
    a.fit(p.data_ptr(), n, epochs=1, batch=batch, lr=1e-30, weight_decay=0.0)
    g = a.grad(p.cpu().numpy())[0]
    b.fit(p.data_ptr(), n, epochs=1, batch=batch, lr=1e-2, weight_decay=0.0)
    w0, w1 = a.get_state()[: len(g)], b.get_state()[: len(g)]
    want = -1e-2 * g / (np.abs(g) + 1e-8)
    big = np.abs(g) > 1e-6   # below, rounding in the sums decides the sign
    assert big.sum() > 1000
    assert np.all(np.abs((w1 - w0) - want)[big] <= 1e-5 + 2e-7 * np.abs(w0[big]))
