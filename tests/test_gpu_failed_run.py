"""A run of a batch that stops on a negative CFL candidate (a cell of negative
width): every other run goes on as without it, also those that its CTA takes
from the queue later."""
import numpy as np
import pytest

from gamma_b200 import gpu, problems

pytestmark = pytest.mark.gpu


def _batch(cells, failing, variant):
    setups = [problems.TubeSetup(ncell=c, vL=.2, vR=.2, pL=12. + .001 * k) for k, c in enumerate(cells)]
    states = [s.initial_state() for s in setups]
    for k in failing:
        states[k].dx[cells[k] // 2] *= -1.
    cfg = gpu.config_cart()
    g = gpu.GammaGPU(cfg, [s.capacity for s in setups])
    g.set_variant(variant)
    pk = problems.pack(states, g.offsets, g.total, cfg.nq)
    g.upload(pk["ntrack"], pk["prim"], pk["x"], pk["dx"], pk["xI"], pk["dt_loc"], pk["t"], pk["it"])
    status = g.step(3)["status"]
    out = g.download()
    res = [problems.unpack(out, r, g.offsets) for r in range(len(cells))]
    g.close()
    return status, np.asarray(out["status"]), res


# 3,000 runs: more than the resident CTAs, each of which takes several; 10: a cluster of CTAs each
@pytest.mark.parametrize("runs,variant", [(3000, 0), (3000, 2), (10, 0)])
def test_other_runs_go_on(gpu_available, runs, variant):
    cells = [60 - (k * 40) // runs for k in range(runs)]  # the queue takes long runs first
    failing = [0, runs // 3]
    st, each, got = _batch(cells, failing, variant)
    ok, none, want = _batch(cells, [], variant)
    assert ok == 0 and not none.any() and st != 0
    assert sorted(np.flatnonzero(each)) == failing and np.all(each[failing] == st)
    for k in range(runs):
        if k in failing:
            assert got[k].it == 1  # stopped after the step that failed
            continue
        assert got[k].it == 3 and got[k].t == want[k].t
        for f in ("prim", "x", "dx", "xI", "dt_loc"):
            assert np.array_equal(getattr(got[k], f), getattr(want[k], f)), (k, f)
