"""The 1D regrid, whose merged cells are formed after the walk, against the C
restatement of the reference's loop, on uneven tracks: runs of merges, merged
cells that are merged again, splits beside merged cells, and merged cells that
turn out high-pressure where neither of their cells was (u != 0: the walk
assumes otherwise and has to be done again)."""
import numpy as np
import pytest

from gamma_b200 import gpu, problems
from oracle import port
from oracle.refsim import Snapshot

pytestmark = pytest.mark.gpu


def _track(seed, n, amp):
    """A BM1D track of n cells with uneven widths and, ahead of the shock,
    velocities of either sign."""
    rng = np.random.default_rng(seed)
    s = problems.Bm1dSetup(eta=1e-10, lorentz_mode=1, lfac_shock2=1e4, ncell=n, nmax=3 * n, grid_log=1, r_lo=.97,
                           r_hi=1.03)
    st = s.initial_state()
    a = slice(2, n + 2)
    w = np.exp(rng.uniform(np.log(.02), np.log(8.), n)) * rng.choice([1., 1., .05], n)
    edge = st.x[2] - st.dx[2] / 2. + np.concatenate([[0.], np.cumsum(w / w.sum())]) * st.dx[a].sum()
    st.x[a], st.dx[a] = .5 * (edge[1:] + edge[:-1]), edge[1:] - edge[:-1]
    ahead = np.zeros(n + 4, bool)
    ahead[a] = st.prim[1, a] < 1.5e-10
    st.prim[1, ahead] = 1.4e-10
    st.prim[2, ahead] = amp * rng.choice([-1., 1.], ahead.sum())
    st.xI[1:n + 2] = edge  # interfaces of the active cells
    problems._update_ghosts(st.prim, st.x, st.dx, st.xI, 2)
    st.dt_loc = np.exp(rng.uniform(0., 5., n + 4))
    return s, st


def _both(seed, n, amp):
    """The regrid on the GPU and by the restated loop."""
    s, st = _track(seed, n, amp)
    g = gpu.GammaGPU(gpu.config_sph(), [s.capacity])
    g.set_params([s.run_params()])
    pk = problems.pack([st], g.offsets, g.total, 10)
    g.upload(pk["ntrack"], pk["prim"], pk["x"], pk["dx"], pk["xI"], pk["dt_loc"], pk["t"], pk["it"])
    stats = g.regrid()
    got = problems.unpack(g.download(), 0, g.offsets)
    g.close()
    ps = port.PortSim(port.bm1d_config(eta=1e-10, lorentz_mode=1, lfac_shock2=1e4, ncell=n, nmax=3 * n, grid_log=1,
                                       r_lo=.97, r_hi=1.03))
    ps.init()
    z = np.zeros(st.ntrack)
    ps.load(Snapshot(t=st.t, dt=0., it=0, ntrack=st.ntrack, prim=st.prim, x=st.x, dx=st.dx, dt_loc=st.dt_loc, sd=z,
                     pspec=z, shocked=z, xI=st.xI))
    ps.regrid()
    want = ps.snapshot()
    # the decisions, exactly
    assert stats["merges"] > 0 and got.ntrack == want.ntrack
    for k in ("x", "dx", "dt_loc", "xI"):
        assert np.array_equal(getattr(got, k), getattr(want, k)), k
    return got, want


SIZES = [(0, 40), (1, 100), (2, 257), (3, 600), (4, 1500)]


@pytest.mark.parametrize("seed,n", SIZES)
def test_merged_cells_match_the_restated_loop(gpu_available, seed, n):
    got, want = _both(seed, n, 0.)
    # merged cells' primitives: two root finders, apart by 1e-13 of p and the noise eps E of a cold cell
    scale = np.abs(want.prim) + 1e-12 * (want.prim[0] * (1. + want.prim[2] ** 2))
    assert np.all(np.abs(got.prim - want.prim) <= 1e-7 * scale)


@pytest.mark.parametrize("seed,n", SIZES)
def test_decisions_when_merging_heats_cells(gpu_available, seed, n):
    """Cells of either velocity merge: the momenta cancel and the energy heats
    the merged cell above the criterion's pressure."""
    got, _ = _both(seed, n, .4)
    assert (got.prim[1] > 1e-3).any()
