"""gamma_mlp_train against the same mini-batches and Adam in 64 bits: the loss of
each epoch and the trained parameters, over batches of less than a tile to the
whole set and over a few epochs."""
import math

import numpy as np
import pytest

from gamma_b200 import gpu
from test_gpu_train_tiles import _grad64

pytestmark = pytest.mark.gpu

H, SEED, LR, LR_FINAL = 64, 7, 3e-3, 1e-4
M64 = (1 << 64) - 1
MULTIPLIERS = (1000003, 999983, 999979, 999961, 999959, 999953, 999931, 999917)


def _inputs(n, seed):
    """Pairs over the network's range (features of gamma_mlp_pairs' uniform
    states), Glorot-uniform weights."""
    rng = np.random.default_rng(seed)
    lfac = np.exp(rng.uniform(0., math.log(1e3), n))
    rho = 10. ** rng.uniform(-6., 6., n)
    p = rho * 10. ** rng.uniform(-10., 3., n)
    D, h = lfac * rho, 1. + 4. * p / rho
    s, tau = h * np.sqrt(lfac * lfac - 1.), h * lfac - p / D - 1.
    x = np.stack([np.log1p(s) / 8., np.log10(np.maximum(tau - (np.sqrt(1. + s * s) - 1.), 1e-30)) / 10.,
                  np.log10(D) / 6.], 1).astype(np.float32)
    y = np.stack([(np.log(p / D) + 14.) / 10., np.log(lfac) / 3.], 1).astype(np.float32)
    glorot = [rng.uniform(-1., 1., k) * math.sqrt(6. / f) for k, f in ((3 * H, 3 + H), (H * H, 2 * H), (2 * H, H + 2))]
    P = np.concatenate([glorot[0], np.zeros(H), glorot[1], np.zeros(H), glorot[2], np.zeros(2)]).astype(np.float32)
    return x, y, P


def _mix(z):
    z = (z + 0x9e3779b97f4a7c15) & M64
    z = ((z ^ (z >> 30)) * 0xbf58476d1ce4e5b9) & M64
    z = ((z ^ (z >> 27)) * 0x94d049bb133111eb) & M64
    return z ^ (z >> 31)


def _train64(P, x, y, batch, epochs):
    n = len(x)
    P, m, v = P.astype(np.float64), np.zeros(P.size), np.zeros(P.size)
    per = -(-n // batch)
    step, losses = 0, []
    for e in range(epochs):
        h = _mix(SEED ^ (0x1234567 + e))
        mul = next((c for c in (MULTIPLIERS[(h + j) % 8] % n for j in range(8)) if c > 0 and math.gcd(c, n) == 1), 1)
        order = (mul * np.arange(n) + h % n) % n
        loss = 0.
        for b in range(per):
            k = order[b * batch:(b + 1) * batch]
            g, l = _grad64(P, x[k], y[k])
            loss += l
            frac = step / (per * epochs - 1) if per * epochs > 1 else 0.
            lr = LR_FINAL + .5 * (LR - LR_FINAL) * (1. + math.cos(math.pi * frac))
            step += 1
            m, v = .9 * m + .1 * g, .999 * v + .001 * g * g
            P = P - lr * (m / (1. - .9 ** step)) / (np.sqrt(v / (1. - .999 ** step)) + 1e-8)
        losses.append(loss / per)
    return P, np.array(losses)


@pytest.mark.parametrize("n,batch,epochs", [(84300, 1000, 1), (20001, 8192, 2), (30001, 997, 2), (5000, 50, 3),
                                            (150007, 150007, 3), (700, 1000, 4), (130, 100, 3)])
def test_training_against_64_bits(gpu_available, n, batch, epochs):
    import torch
    x, y, P0 = _inputs(n, n)
    dx, dy, P = (torch.tensor(a, device="cuda") for a in (x, y, P0))
    loss = gpu.mlp_train(P.data_ptr(), dx.data_ptr(), dy.data_ptr(), n, epochs=epochs, batch=batch, lr=LR,
                         lr_final=LR_FINAL, seed=SEED)
    want, wl = _train64(P0, x, y, batch, epochs)
    # the same training with each operation rounded to 32 bits, in plain numpy: loss
    # within 1.3e-7 (half of it the rounding of the result), parameters within
    # 4.4e-7 in norm; twice that, for __expf's few ulp
    assert np.abs(loss / wl - 1.).max() <= 3e-7
    assert np.linalg.norm(P.cpu().numpy() - want) <= 1e-6 * np.linalg.norm(want)
