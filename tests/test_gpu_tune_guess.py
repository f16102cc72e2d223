"""The autotuner with a learned guess set: the first step after set_guess, which
runs with the network whatever the warm starts, counts for no launch shape."""
import pytest

from gamma_b200 import gpu, problems

pytestmark = pytest.mark.gpu


def test_first_learned_step_is_not_timed(gpu_available):
    import torch
    # more runs than 16 per SM, so that the default shape is one CTA of 128 threads per run
    setups = [problems.TubeSetup(ncell=400 + k % 300, pL=12. + .001 * k) for k in range(2600)]
    states = [s.initial_state() for s in setups]
    g = gpu.GammaGPU(gpu.config_cart(), [s.capacity for s in setups])
    pk = problems.pack(states, g.offsets, g.total, 6)
    g.upload(pk["ntrack"], pk["prim"], pk["x"], pk["dx"], pk["xI"], pk["dt_loc"], pk["t"], pk["it"])
    P = torch.zeros(gpu.mlp_param_count(), dtype=torch.float32, device="cuda")
    gpu.mlp_init(P.data_ptr(), 5)
    torch.cuda.synchronize()
    plain, learned = [], []
    for _ in range(5):
        g.set_guess(0)
        plain.append(g.autotune(1)[0][0])
        g.set_guess(P.data_ptr())
        learned.append(g.autotune(1)[0][0])
    g.close()
    # the network's step takes twice the plain one; the plain one behind the policy 1% more
    assert min(learned) <= 1.3 * min(plain), (plain, learned)
