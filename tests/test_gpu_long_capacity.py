"""Contexts of few runs with a long track's capacity: the regrid's bit words take
shared memory from the step kernel, so the default launch shape has to be one that
still fits, up to the capacity that 128 threads leave room for.  The capacity does
not enter the arithmetic: the same bits as with a short one."""
import numpy as np
import pytest

from gamma_b200 import gpu, problems

pytestmark = pytest.mark.gpu

KW = dict(eta=1e-10, lorentz_mode=1, lfac_shock2=1e4, grid_log=1, r_lo=.97, r_hi=1.03)


def _steps(caps, state, setup, guess=None):
    """Three steps of the same run in every track; the first track."""
    g = gpu.GammaGPU(gpu.config_sph(), caps)
    g.set_params([setup.run_params()] * len(caps))
    if guess is not None:
        g.set_guess(guess.data_ptr())
    pk = problems.pack([state] * len(caps), g.offsets, g.total, 10)
    g.upload(pk["ntrack"], pk["prim"], pk["x"], pk["dx"], pk["xI"], pk["dt_loc"], pk["t"], pk["it"])
    assert g.step(3)["status"] == 0
    out = problems.unpack(g.download(), 0, g.offsets)
    g.close()
    return out


# 128 threads with four rows of words fit up to 389,632 cells; 512 up to 175,744, 256
# (which batches of 444 runs and more take) up to 319,232
@pytest.mark.parametrize("learned", [False, True])
@pytest.mark.parametrize("cap,runs", [(175744, 1), (175745, 1), (300000, 1), (319233, 1), (300000, 600)])
def test_default_shape_fits(gpu_available, cap, runs, learned):
    import torch
    s = problems.Bm1dSetup(ncell=200, nmax=600, **KW)
    guess = None
    if learned:
        guess = torch.zeros(gpu.mlp_param_count(), dtype=torch.float32, device="cuda")
        gpu.mlp_init(guess.data_ptr(), 3)
        torch.cuda.synchronize()
    st = s.initial_state()
    got = _steps([cap] + [s.capacity] * (runs - 1), st, s, guess)
    want = _steps([s.capacity], st, s)
    assert got.ntrack == want.ntrack
    if not learned:  # (with the guess the roots are the same to the search's tolerance)
        for k in ("prim", "x", "dx", "xI", "dt_loc"):
            assert np.array_equal(getattr(got, k), getattr(want, k)), k


def test_largest_capacity(gpu_available):
    s = problems.Bm1dSetup(ncell=200, nmax=600, **KW)
    assert _steps([389632], s.initial_state(), s).ntrack > 0
