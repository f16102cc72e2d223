"""Device memory of a refining 1D context: 642 bytes per cell of capacity
(the state, the step's and the regrid's arrays), which decides the largest batch
that a GPU takes."""
import pytest

from gamma_b200 import gpu

pytestmark = pytest.mark.gpu


def test_bytes_per_cell(gpu_available):
    import torch
    torch.zeros(1, device="cuda")
    gpu.GammaGPU(gpu.config_sph(), [1000]).close()  # the kernels are loaded
    free = torch.cuda.mem_get_info()[0]
    g = gpu.GammaGPU(gpu.config_sph(), [4000] * 1000)
    used = free - torch.cuda.mem_get_info()[0]
    cells = g.total
    g.close()
    assert used <= 642 * cells + 2 ** 20 * 48  # 24 arrays, each rounded up to 2 MiB
