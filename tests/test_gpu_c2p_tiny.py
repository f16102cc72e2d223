"""cons2prim of states whose squares underflow: where f(p_lo) < 0 there is no
solution, and the pressure stays the starting one (rel_sph.cpp:243-286), also
where E^2 - S^2 and D^2 have lost their digits."""
import numpy as np
import pytest

from gamma_b200 import gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sph", [False, True])
@pytest.mark.parametrize("decade", [-140, -155, -156, -158, -160])
def test_no_solution_below_the_squares_range(gpu_available, sph, decade):
    import torch
    rng = np.random.default_rng(-decade)
    n = 40000
    E = 10. ** (decade + rng.uniform(-1., 1., n))
    S = E * rng.uniform(0., 1., n)
    D = np.sqrt(E - S) * np.sqrt(E + S) * (1. + rng.choice([0., 1e-3, 1e-2], n) * rng.uniform(-1., 1., n))
    tau = E - D
    E, S = D + tau, np.sqrt(S * S)
    with np.errstate(divide="ignore", invalid="ignore"):
        arg = 1. - (S * S) / (E * E)
        lfac = 1. / np.sqrt(np.abs(arg) if sph else arg)
        f = E - D * lfac - 0. * lfac * lfac  # f(0) as the search forms it (NaN where lfac is infinite)
    none = (f < 0.) & (S * (1. + 1e-13) < E)
    assert none.sum() > 1000
    cfg = gpu.config_sph() if sph else gpu.config_cart()
    cons, prim = np.zeros((cfg.nq, n)), np.ones((cfg.nq, n))
    cons[0], cons[1], cons[2] = D, tau, S
    dc, dp = torch.tensor(cons, device="cuda"), torch.tensor(prim, device="cuda")
    gpu.cons2prim_device(cfg, dc.data_ptr(), dp.data_ptr(), n)
    torch.cuda.synchronize()
    assert np.all(dp.cpu().numpy()[1, none] == 1.)
