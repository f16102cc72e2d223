"""The training kernels' tiles of 64 samples: gradient and loss at sample counts
around a tile and around one tile per SM, against the same formulas in 64 bits,
and training that repeats bit for bit."""
import numpy as np
import pytest

from gamma_b200 import gpu

pytestmark = pytest.mark.gpu

H = 64


def _params(seed):
    rng = np.random.default_rng(seed)
    return np.concatenate([rng.normal(0., .5, 3 * H), rng.normal(0., .3, H), rng.normal(0., .15, H * H),
                           rng.normal(0., .2, H), rng.normal(0., .2, 2 * H), rng.normal(0., .1, 2)]).astype(np.float32)


def _grad64(P, x, y):
    cut = np.cumsum([0, 3 * H, H, H * H, H, 2 * H, 2])
    W1, b1, W2, b2, W3, b3 = (P[i:j].astype(np.float64) for i, j in zip(cut[:-1], cut[1:]))
    W1, W2, W3 = W1.reshape(H, 3), W2.reshape(H, H), W3.reshape(2, H)
    x, y = x.astype(np.float64), y.astype(np.float64)
    z1 = x @ W1.T + b1
    s1 = 1. / (1. + np.exp(-z1))
    z2 = (z1 * s1) @ W2.T + b2
    s2 = 1. / (1. + np.exp(-z2))
    r = (z2 * s2) @ W3.T + b3 - y
    d3 = r / len(x)
    d2 = (d3 @ W3) * (s2 + z2 * s2 * (1. - s2))
    d1 = (d2 @ W2) * (s1 + z1 * s1 * (1. - s1))
    return np.concatenate([(d1.T @ x).ravel(), d1.sum(0), (d2.T @ (z1 * s1)).ravel(), d2.sum(0),
                           (d3.T @ (z2 * s2)).ravel(), d3.sum(0)]), .5 * (r * r).sum() / len(x)


@pytest.mark.parametrize("n", [1, 2, 63, 64, 65, 129, 9471, 9472, 9473, 30000])
def test_gradient_at_tile_edges(gpu_available, n):
    import torch
    rng = np.random.default_rng(n)
    P, x, y = _params(1), rng.normal(0., 1., (n, 3)).astype(np.float32), rng.normal(0., 1., (n, 2)).astype(np.float32)
    d = [torch.tensor(a, device="cuda") for a in (P, x, y)]
    g, loss = torch.full((P.size,), 7., device="cuda"), torch.full((1,), 7., device="cuda")
    gpu.mlp_loss_grad(d[0].data_ptr(), d[1].data_ptr(), d[2].data_ptr(), n, g.data_ptr(), loss.data_ptr())
    torch.cuda.synchronize()
    want, wl = _grad64(P, x, y)
    # FP32 sums of n terms, and __expf's few ulp: 2^-24 sqrt(n) and 1e-6 of the largest gradient, with room
    tol = (1e-5 + 1e-6 * np.sqrt(n)) * np.abs(want).max()
    assert np.abs(g.cpu().numpy() - want).max() <= tol
    assert abs(loss.item() - wl) <= (1e-5 + 1e-6 * np.sqrt(n)) * wl


@pytest.mark.parametrize("n,batch", [(5000, 64), (5000, 1000), (20001, 8192), (30000, 30000)])
def test_training_repeats_bit_for_bit(gpu_available, n, batch):
    import torch
    rng = np.random.default_rng(2)
    x = torch.tensor(rng.normal(0., 1., (n, 3)).astype(np.float32), device="cuda")
    y = torch.tensor(rng.normal(0., 1., (n, 2)).astype(np.float32), device="cuda")
    got = []
    for _ in range(2):
        P = torch.tensor(_params(3), device="cuda")
        loss = gpu.mlp_train(P.data_ptr(), x.data_ptr(), y.data_ptr(), n, epochs=2, batch=batch)
        got.append((P.cpu().numpy(), loss))
    assert np.array_equal(got[0][0], got[1][0]) and np.array_equal(got[0][1], got[1][1])
    assert got[0][1][1] < got[0][1][0]  # and it learns
