"""One run over a cluster of CTAs (few runs) against one CTA per run (a batch of
more runs than half the SMs): the same bits, for track lengths at and around
the edges of the CTAs' segments, in several launch shapes, with and without a
regrid."""
import numpy as np
import pytest

from gamma_b200 import gpu, problems

pytestmark = pytest.mark.gpu

FILL = 150  # runs of a batch that takes one CTA each


def _run(cfg, setups, states, steps, variant, params=False):
    g = gpu.GammaGPU(cfg, [s.capacity for s in setups])
    if params:
        g.set_params([s.run_params() for s in setups])
    g.set_variant(variant)
    pk = problems.pack(states, g.offsets, g.total, cfg.nq)
    g.upload(pk["ntrack"], pk["prim"], pk["x"], pk["dx"], pk["xI"], pk["dt_loc"], pk["t"], pk["it"])
    assert g.step(steps)["status"] == 0
    out = g.download()
    res = [problems.unpack(out, r, g.offsets) for r in range(len(setups))]
    g.close()
    return res


def _same(a, b):
    assert a.ntrack == b.ntrack and a.t == b.t and a.it == b.it
    for k in ("prim", "x", "dx", "xI", "dt_loc"):
        assert np.array_equal(getattr(a, k), getattr(b, k), equal_nan=True), k


@pytest.mark.parametrize("variant,timestep", [(0, gpu.TS_RK3), (1, gpu.TS_RK3), (2, gpu.TS_RK3), (4, gpu.TS_RK3),
                                              (0, gpu.TS_EULER)])
def test_tubes_alone_and_in_a_batch(gpu_available, variant, timestep):
    # ntrack = ncell + 4; segments end at 64 c - 1, 128 c - 1, 256 c - 1, 512 c - 1 cells past the first
    cells = [3, 4, 59, 60, 61, 62, 123, 124, 125, 126, 187, 251, 252, 253, 254, 379, 507, 508, 1019, 1020, 1021, 2043,
             4091, 4093]
    setups = [problems.TubeSetup(ncell=c, vL=.3 - .01 * k, vR=.3 - .01 * k, pL=12. + .1 * k)
              for k, c in enumerate(cells)]
    setups += [problems.TubeSetup(ncell=20)] * (FILL - len(setups))
    states = [s.initial_state() for s in setups]
    cfg = gpu.config_cart(timestep=timestep)
    batch = _run(cfg, setups, states, 4, variant)
    for k in range(len(cells)):  # one run: a cluster of up to 8 CTAs
        _same(_run(cfg, setups[k:k + 1], states[k:k + 1], 4, variant)[0], batch[k])
    for a, b in zip(_run(cfg, setups[:len(cells)], states[:len(cells)], 4, variant), batch):  # clusters of up to 4
        _same(a, b)


@pytest.mark.parametrize("variant", [0, 1, 2, 6])
def test_blast_waves_alone_and_in_a_batch(gpu_available, variant):
    kw = dict(eta=1e-10, lorentz_mode=1, lfac_shock2=1e4, grid_log=1, r_lo=.9, r_hi=1.1)
    setups = [problems.Bm1dSetup(ncell=n, nmax=2 * n, Etot=10. ** (51. + .3 * k), **kw)
              for k, n in enumerate([120, 251, 509, 900, 1500])]
    setups += [problems.Bm1dSetup(ncell=40, nmax=80, **kw)] * (FILL - len(setups))
    states = [s.initial_state() for s in setups]
    cfg = gpu.config_sph()
    batch = _run(cfg, setups, states, 12, variant, params=True)
    assert any(b.ntrack != s.ntrack for b, s in zip(batch, states))  # the regrid acted
    for k in range(5):
        _same(_run(cfg, setups[k:k + 1], states[k:k + 1], 12, variant, params=True)[0], batch[k])
