"""A merged cell that the 1D regrid's walk has to form before it goes on, and
that turns out high-pressure where neither of its cells was: the shock index, and
with it the decisions of the cells behind, follow it as in the restated loop."""
import numpy as np
import pytest

import test_gpu_regrid_walk as walk
from gamma_b200 import problems

pytestmark = pytest.mark.gpu

NARROW, PLAIN, WIDE = .05, .5, 4.  # widths in units of rOut dth: merged; split only in the shock's window; split


def _track(c, nxt):
    """Gas at rest, of PLAIN cells, in which cell c merges with the cell on its
    right, of the opposite momentum; nxt: the width of the cell after those."""
    n = 120
    s = problems.Bm1dSetup(eta=1e-10, lorentz_mode=1, lfac_shock2=1e4, ncell=n, nmax=3 * n, grid_log=1, r_lo=.97,
                           r_hi=1.03)
    st = s.initial_state()
    w = np.full(n, PLAIN)
    w[:12] = .2  # the window of the first cell, the shock where no cell is marked
    w[c], w[c + 1], w[c + 2] = NARROW, .3, nxt
    rout = st.x[n + 1]
    w *= rout * s.dth
    edge = rout + w[-1] / 2. - np.concatenate([[0.], np.cumsum(w[::-1])])[::-1]
    a = slice(2, n + 2)
    st.prim[:, a] = st.prim[:, n + 1:n + 2]  # the ambient gas
    st.x[a], st.dx[a] = .5 * (edge[1:] + edge[:-1]), edge[1:] - edge[:-1]
    st.xI[1:n + 2] = edge
    st.prim[2, 2 + c], st.prim[2, 3 + c] = .03, -.005
    if nxt == NARROW:  # a marked cell that merges with the merged one, on its left
        st.prim[1, 4 + c] = 2e-10
    problems._update_ghosts(st.prim, st.x, st.dx, st.xI, 2)
    return s, st


@pytest.mark.parametrize("nxt", [WIDE, NARROW])
@pytest.mark.parametrize("c", [14, 27, 28, 29, 60, 90])
def test_marks_of_cells_formed_in_the_walk(gpu_available, monkeypatch, c, nxt):
    monkeypatch.setattr(walk, "_track", lambda *_: _track(c, nxt))
    got, want = walk._both(0, 120, 0.)
    assert want.ntrack > 125 and (got.prim[1] > 1e-6).any()  # split behind the heated cell
