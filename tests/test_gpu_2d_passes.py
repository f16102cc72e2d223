"""How the 2D step's passes divide the cells does not show in their results.

Every value of a cell or an interface is formed by the same operations in the
same order wherever the cell lies in a pass's tiles, with any share of the
transverse gradients' slots per thread, from a track index formed in one launch
or two, from either place of the two grad_f1 arrays, and from a graph or direct
launches.  So the live cells of equal runs agree bit for bit: nothing here has
a tolerance.
"""
import numpy as np
import pytest

from gamma_b200 import gpu2d, problems

pytestmark = pytest.mark.gpu


def _grid(s, first=0, n=None):
    """A context on the tracks first .. first+n-1 of the setup, uploaded."""
    n = s.ntheta if n is None else n
    th, dth = s.theta()
    st, gh = s.initial_state(), s.ngst
    cut = slice(first * st.cap, (first + n + 2 * gh) * st.cap)
    st.prim, st.x, st.dx, st.xI = (a[..., cut].copy() for a in (st.prim, st.x, st.dx, st.xI))
    st.ntrack, st.NJ = st.ntrack[first:first + n + 2 * gh].copy(), n + 2 * gh
    if first:  # the leading ghost tracks are filled on the device
        for a in (st.prim, st.x, st.dx, st.xI):
            a[..., :gh * st.cap] = 0.
    g = gpu2d.Grid2DGPU(n, s.nmax, th[first:first + n], dth[first:first + n])
    g.set_params(s.params())
    g.upload(st, run_ghosts=True)
    return g


def _live(g):
    st = g.download()
    assert int(st.extra["status"][0]) == 0
    out = [np.array([st.t, float(st.it)]), st.ntrack.astype(np.float64)]
    for j in range(st.NJ):
        o, n = j * st.cap, int(st.ntrack[j])
        out += [a[..., o:o + n].ravel() for a in (st.prim, st.x, st.dx, st.dt_loc, st.grad_mv, st.grad_f1)]
        out.append(st.xI[o:o + n - 1])
    return np.concatenate(out)


def _same(a, b):
    assert a.shape == b.shape and np.array_equal(a, b, equal_nan=True)


@pytest.mark.parametrize("ncell", [57, 61, 200])
def test_capacity_and_steps_per_call(gpu_available, ncell):
    """12 + 4 tracks whose capacity takes the grid past 128 and 1,024 cells per
    SM of 148 (5, 2 and 1 threads per cell in the transverse gradients)."""
    runs = []
    for nmax, calls, graphs in ((ncell + 100, (6,), True), (3000, (1, 2, 3), True), (12000, (4, 1, 1), False)):
        s = problems.Jet2dSetup(ncell=ncell, ntheta=12, nmax=nmax, merge_DR_slow=.3)
        g = _grid(s)
        g.use_graphs(graphs)
        g.prepare_stage(2)  # leaves the arrays in their other places
        g.close()
        g = _grid(s)
        g.use_graphs(graphs)
        for k in calls:
            assert g.step(k)["status"] == 0
        runs.append(_live(g))
        g.close()
    _same(runs[0], runs[1])
    _same(runs[0], runs[2])


def test_a_stage_left_in_the_middle(gpu_available):
    """The diagnostics stop within a step, with the arrays in either place; an
    upload starts anew from there, also with the graphs captured before."""
    s = problems.Jet2dSetup(ncell=80, ntheta=6, nmax=200)
    g = _grid(s)
    first = g.download()
    g.step(3)
    want = _live(g)
    for stage in (1, 2, 3, 2):
        g.prepare_stage(stage)
        g.upload(first)
        g.step(3)
        _same(want, _live(g))
    g.close()


@pytest.mark.parametrize("ntheta, ncell, first, n", [(20, 57, 3, 14), (20, 61, 1, 19), (20, 8, 5, 12), (9, 700, 2, 7),
                                                     (11000, 8, 700, 2000)])
def test_stage_of_some_tracks_alone(gpu_available, ntheta, ncell, first, n):
    """Stage-1 fluxes of tracks four or more from the ends of a part of the
    tracks: the part's cells lie elsewhere in the tiles, and with 11,000 tracks
    the whole's index takes its two launches."""
    s = problems.Jet2dSetup(ncell=ncell, ntheta=ntheta, nmax=ncell + 8)
    whole, part = _grid(s), _grid(s, first, n)
    got = []
    for g, off in ((whole, first), (part, 0)):
        g.prepare_stage(1)
        nt, cap = g.download().ntrack, g.cap
        f = g.download_fluxes()
        rows = []
        for j in range(2 + 4, 2 + n - 4) if n > 8 else range(2 + 3, 2 + n - 3):
            o, m = (j + off) * cap, int(nt[j + off])
            for k in ("flux", "v", "lL", "lR"):
                rows.append(f[k][..., o:o + m - 1].ravel())
            for k in ("f1lo", "f1hi", "grad_f1"):
                rows.append(f[k][..., o:o + m].ravel())
        got.append(np.concatenate(rows))
        g.close()
    assert np.count_nonzero(got[0]) > 0
    _same(got[0], got[1])
