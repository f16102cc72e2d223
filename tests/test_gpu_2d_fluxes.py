"""gamma_2d_download_fluxes after whole steps returns what the fluxes of their
last stage returned, each theta side by itself, from a graph or direct launches,
and leaves the state as it is."""
import numpy as np
import pytest

from gamma_b200 import gpu, gpu2d, problems

pytestmark = pytest.mark.gpu


def _grid(s, timestep):
    th, dth = s.theta()
    g = gpu2d.Grid2DGPU(s.ntheta, s.nmax, th, dth, timestep=timestep)
    g.set_params(s.params())
    g.upload(s.initial_state(), run_ghosts=True)
    return g


def _fluxes(g, ntrack):
    f, out = g.download_fluxes(), []
    for j, n in enumerate(ntrack):
        o = j * g.cap
        out += [f[k][..., o:o + n - 1].ravel() for k in ("v", "lL", "lR", "flux")]
        out += [f[k][..., o:o + n].ravel() for k in ("f1lo", "f1hi", "grad_f1")]
    return np.concatenate(out)


@pytest.mark.parametrize("steps", [1, 2, 3])
@pytest.mark.parametrize("timestep,graphs", [(gpu.TS_RK3, True), (gpu.TS_RK3, False), (gpu.TS_EULER, True)])
def test_fluxes_after_steps(gpu_available, steps, timestep, graphs):
    s = problems.Jet2dSetup(ncell=60, ntheta=6, nmax=200)
    a, b = _grid(s, timestep), _grid(s, timestep)
    first = a.download()
    a.use_graphs(graphs)
    if steps > 1:
        b.step(steps - 1)
    b.prepare_stage(3 if timestep == gpu.TS_RK3 else 1)  # the last stage, up to its fluxes
    nt = b.download().ntrack
    want = _fluxes(b, nt)
    a.step(steps)
    assert np.array_equal(a.download().ntrack, nt)
    before = a.download()
    assert np.count_nonzero(want) > 0
    for _ in range(2):
        assert np.array_equal(_fluxes(a, nt), want, equal_nan=True)
    after = a.download()
    for k in ("prim", "x", "dx", "xI", "dt_loc", "grad_mv", "grad_f1", "nbr"):
        assert np.array_equal(getattr(after, k), getattr(before, k), equal_nan=True), k
    for k in ("sd", "pspec", "shocked"):
        assert np.array_equal(after.extra[k], before.extra[k], equal_nan=True), k
    a.upload(first)
    assert np.array_equal(_fluxes(a, nt), want, equal_nan=True)  # the last stage's, still
    b.close()
    a.step(steps)
    assert np.array_equal(_fluxes(a, nt), want, equal_nan=True)  # and again, from the other side
    a.step(1)
    a.upload(first)
    a.step(steps - 1)
    a.prepare_stage(3 if timestep == gpu.TS_RK3 else 1)
    a.upload(first)
    assert np.array_equal(_fluxes(a, nt), want, equal_nan=True)
    a.close()
