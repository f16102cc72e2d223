"""A step of the 2D context whose graph cannot be captured (its stream is already
being captured, an error on the host) leaves the context as it was."""
import ctypes

import pytest

from gamma_b200 import gpu, problems
from test_gpu_2d_passes import _grid, _live, _same

pytestmark = pytest.mark.gpu

RELAXED = 2  # CU_STREAM_CAPTURE_MODE_RELAXED


def _failing_step(g, nsteps):
    cu = ctypes.CDLL("libcuda.so.1")
    stream = ctypes.c_void_p(g.stream)
    graph = ctypes.c_void_p()
    assert cu.cuStreamBeginCapture_v2(stream, RELAXED) == 0
    with pytest.raises(gpu.GammaError):
        g.step(nsteps, stats=False)
    cu.cuStreamEndCapture(stream, ctypes.byref(graph))
    if graph:
        cu.cuGraphDestroy(graph)


@pytest.mark.parametrize("captured", [0, 1])
def test_step_after_a_failed_capture(gpu_available, captured):
    """captured: 1, the graph of one place of the two grad_f1 arrays is there
    and that of the other fails."""
    s = problems.Jet2dSetup(ncell=60, ntheta=6, nmax=200)
    runs = []
    for fails in (False, True):
        g = _grid(s)
        if captured:
            g.step(1)
            g.prepare_stage(2)  # the arrays back in the places of that step's start
        if fails:
            _failing_step(g, 2)
        g.step(1)
        runs.append(_live(g))
        g.step(3)
        runs.append(_live(g))
        g.close()
    _same(runs[0], runs[2])
    _same(runs[1], runs[3])
