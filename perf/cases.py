"""Workloads of the moving-mesh step, its primitive recovery and its network.

Each case is one job as a user's program runs it through the public entry
points: a state or snapshot in pinned host memory is uploaded, some steps are
taken, and the new snapshot is downloaded; or a batch of conserved states on
the device is recovered; or a network is trained.  ``listed`` names twelve of
them, ``draw`` gives others of the same ranges.

Sizes and options: the shock tubes, the Blandford-McKee runs and the wedge of
theta tracks of the benchmark and the tests, from a single short run (bound by
latency and launches) up to thousands of runs at once.
"""
import ctypes
import math

import numpy as np
import torch

from gamma_b200 import gpu, gpu2d, problems

# ---------------------------------------------------------------------------
# cases


def listed():
    return [
        # one short planar tube, stepped one call at a time with its statistics read back,
        # as the loop of Simu::run drives it: latency of the smallest call
        dict(name="tube_one", kind="tubes", runs=1, lo=500, hi=500, steps=10, per_call=1, stats=True,
             hydro="cart", timestep="rk3", tune=False),
        # a handful of long tubes in one call of many steps (fewer runs than SMs)
        dict(name="tubes_few", kind="tubes", runs=12, lo=1001, hi=8191, steps=20, per_call=20, stats=True,
             hydro="cart", timestep="rk3", tune=False),
        # the headline batch: thousands of uneven tubes, one step a launch, tuned launch shape
        dict(name="tubes_many", kind="tubes", runs=4096, lo=256, hi=8192, steps=20, per_call=1, stats=False,
             hydro="cart", timestep="rk3", tune=True),
        # tubes in arrays that the caller owns (its own memory pool), ragged sizes
        dict(name="tubes_pool", kind="pool", runs=200, lo=257, hi=8191, steps=2, timestep="rk3"),
        # the other hydro module and time stepping: cylindrical, Euler
        dict(name="tubes_cyl_euler", kind="tubes", runs=600, lo=256, hi=4096, steps=20, per_call=1, stats=False,
             hydro="cyl", timestep="euler", tune=False),
        # one Blandford-McKee blast wave of 2,000 log cells, regrid, shocks and tracers on
        dict(name="blast_one", kind="blast", runs=1, lo=2000, hi=2000, settle=10, steps=50, per_call=50,
             tune=False),
        # the first steps of a parameter sweep: the regrid merges most of the ambient cells
        dict(name="blast_start", kind="blast", runs=256, lo=1000, hi=8000, settle=0, steps=3, per_call=1, tune=False),
        # the settled sweep: 1,024 uneven runs, tuned launch shape
        dict(name="blast_sweep", kind="blast", runs=1024, lo=1000, hi=8000, settle=8, steps=40, per_call=1,
             tune=True),
        # a thin 2D wedge (launch-bound) and the 512-track jet
        dict(name="wedge", kind="jet", ntheta=16, ncell=400, settle=3, steps=10),
        dict(name="jet", kind="jet", ntheta=512, ncell=4000, settle=3, steps=10),
        # primitive recovery of independent states from p = 1, and started from the network
        dict(name="c2p_cold", kind="c2p", n=4194307, hydro="sph", start="cold"),
        # one epoch of training on the pairs of a run
        dict(name="train", kind="train", n=1000003, epochs=1, batch=8192),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["tubes", "tubes", "pool", "blast", "blast", "jet", "c2p", "c2p", "train"])
    if kind == "tubes":
        runs = _log(rng, 1, 2000)
        lo = _log(rng, 64, 1500)
        hydro = rng.choice(["cart", "cart", "cyl"])
        steps = rng.randint(3, 20)
        return dict(kind=kind, runs=runs, lo=lo, hi=min(8192, lo * rng.randint(1, 16)), steps=steps,
                    per_call=rng.choice([1, steps]), stats=rng.random() < 0.5, hydro=hydro,
                    timestep=rng.choice(["rk3", "rk3", "euler"]), tune=False)
    if kind == "pool":
        return dict(kind=kind, runs=_log(rng, 2, 300), lo=129, hi=rng.randint(300, 4000), steps=rng.randint(1, 3),
                    timestep=rng.choice(["rk3", "euler"]))
    if kind == "blast":
        settle = rng.choice([0, 8])
        steps = rng.randint(2, 20)
        return dict(kind=kind, runs=_log(rng, 1, 400), lo=1000, hi=rng.randint(1001, 8000), settle=settle,
                    steps=steps if settle else min(steps, 4), per_call=rng.choice([1, steps]) if settle else 1,
                    tune=False)
    if kind == "jet":
        return dict(kind=kind, ntheta=_log(rng, 5, 200), ncell=_log(rng, 100, 3000), settle=3,
                    steps=rng.randint(3, 10))
    if kind == "c2p":
        return dict(kind=kind, n=_log(rng, 1000, 4000000), hydro=rng.choice(["sph", "cart"]),
                    start=rng.choice(["cold", "warm", "learned"]))
    return dict(kind=kind, n=_log(rng, 20000, 900000), epochs=rng.randint(1, 2),
                batch=rng.choice([1000, 4096, 8192]))


def prepare(case, seed):
    return _KINDS[case["kind"]][0](case, seed)


def run(state):
    return state.run()


def work(case):
    return _KINDS[case["kind"]][1](case)


def exact(case, seed):
    f = _KINDS[case["kind"]][2]
    return f(case, seed) if f else None


def _sizes(case):
    """Cells of each run: log-uniform over [lo, hi], the same for every seed."""
    rng = np.random.default_rng(12345 + case["runs"])
    return np.exp(rng.uniform(math.log(case["lo"]), math.log(case["hi"]), case["runs"])).round().astype(int)


def _pinned(*shape):
    return torch.zeros(shape, dtype=torch.float64, pin_memory=True)


def _blank(arr, offsets, cap, start, ntrack):
    """Zero the slots past each run's cells that a job may have used (start: the
    cells it began with): a snapshot holds live cells only."""
    for o, c, s, n in zip(offsets, cap, start, ntrack):
        end = min(int(c), max(int(s), int(n)) + 256)
        if n < end:
            arr[:, o + n:o + end] = 0.


# ---------------------------------------------------------------------------
# planar shock tubes


def _tube_states(case, seed, tracks):
    """Initial state of each tube: 1DST-style left and right states, varied."""
    rng = np.random.default_rng(seed)
    out = []
    for n in tracks:
        v = float(rng.uniform(-.5, .5))
        out.append(problems.TubeSetup(ncell=int(n), rhoL=10. * (1. + .2 * float(rng.uniform(-1, 1))),
                                      pL=13.33 * (1. + .2 * float(rng.uniform(-1, 1))), vL=v, vR=v,
                                      xmin=.1 if case.get("hydro") == "cyl" else 0.,
                                      xmax=1.1 if case.get("hydro") == "cyl" else 1.,
                                      xmid=.6 if case.get("hydro") == "cyl" else .5).initial_state())
    return out


def _tube_cfg(case):
    ts = gpu.TS_EULER if case["timestep"] == "euler" else gpu.TS_RK3
    return gpu.config_cyl(timestep=ts) if case.get("hydro") == "cyl" else gpu.config_cart(timestep=ts)


class _Job1D:
    """Upload of a snapshot, steps, download of the new one, for any number of runs."""

    def __init__(self, cfg, caps, case, params=None):
        self.g = gpu.GammaGPU(cfg, caps)
        self.case = case
        if params is not None:
            self.g.set_params(params)
        N = self.g.total
        self.host = {k: _pinned(*s) for k, s in (("prim", (cfg.nq, N)), ("x", (1, N)), ("dx", (1, N)),
                                                 ("dt_loc", (1, N)), ("xI", (1, N)))}
        self.out = {k: _pinned(*v.shape) for k, v in self.host.items()}

    def fill(self, states):
        np_ = {k: v.numpy() for k, v in self.host.items()}
        np_["dt_loc"][:] = problems.DT_INF
        for s, o in zip(states, self.g.offsets):
            n = s.ntrack
            np_["prim"][:, o:o + n] = s.prim
            np_["x"][0, o:o + n] = s.x
            np_["dx"][0, o:o + n] = s.dx
            np_["dt_loc"][0, o:o + n] = s.dt_loc
            np_["xI"][0, o:o + n - 1] = s.xI
        self.ntrack = np.array([s.ntrack for s in states], np.int32)
        self.t = np.array([s.t for s in states])
        self.it = np.array([s.it for s in states], np.int64)
        self.upload()
        if self.case["tune"]:
            self.g.autotune(2)

    def upload(self):
        h = self.host
        self.g.upload_ptrs(self.ntrack, self.t, self.it, h["prim"].data_ptr(), h["x"].data_ptr(),
                           h["dx"].data_ptr(), h["dt_loc"].data_ptr(), h["xI"].data_ptr())

    def run(self):
        self.upload()
        per = self.case["per_call"]
        done = 0
        while done < self.case["steps"]:
            k = min(per, self.case["steps"] - done)
            self.g.step(k, stats=self.case.get("stats", False))
            done += k
        o = self.out
        nt = self.g.download_ptrs(o["prim"].data_ptr(), o["x"].data_ptr(), o["dx"].data_ptr(),
                                  o["dt_loc"].data_ptr(), o["xI"].data_ptr())
        offs, cap = self.g.offsets, (self.g.cap + 1) & ~1
        for k, v in o.items():
            _blank(v.numpy(), offs, cap, self.ntrack, nt - 1 if k == "xI" else nt)
        return {"ntrack": nt, **o}

    def __del__(self):
        self.g.close()


def _tubes(case, seed):
    states = _tube_states(case, seed, _sizes(case))
    job = _Job1D(_tube_cfg(case), [s.ntrack for s in states], case)
    job.fill(states)
    return job


# per zone and step: the state (primitives, x, dx, dt_loc, xI) read and written;
# floating-point operations of the three stages (a division or root as one)
def _tubes_work(case):
    zones = int(_sizes(case).sum()) * case["steps"]
    stages = 1 if case["timestep"] == "euler" else 3
    return {"bytes": 2. * 8 * 9 * zones, "flops": 550. * stages * zones}


# ---------------------------------------------------------------------------
# tubes in the caller's own device arrays


class _Pool:
    def __init__(self, case, seed):
        sizes = _sizes(case) + 4
        # the entry point's fixed workspace bounds a call to 690,000 cells
        keep = np.cumsum((sizes + 1) & ~1) <= 680000
        sizes = sizes[keep]
        states = _tube_states(case, seed, sizes - 4)
        offs = np.concatenate([[0], np.cumsum((sizes + 1) & ~1)])
        pk = problems.pack(states, offs[:-1], int(offs[-1]), 6)
        dev = torch.device("cuda")
        self.total, self.runs, self.case, self.cfg = int(offs[-1]), len(states), case, _tube_cfg(case)
        rs = np.zeros(self.runs, dtype=[("ntrack", "i4"), ("status", "i4"), ("t", "f8"), ("dt", "f8"), ("it", "i8")])
        rs["ntrack"] = pk["ntrack"]
        # the primitive rows as the entry point stores them: slot 3 (zero in 1D) is left out
        prim = np.ascontiguousarray(pk["prim"][[0, 1, 2, 4, 5]])
        self.first = [torch.tensor(a, device=dev) for a in (prim, pk["x"], pk["dx"], pk["dt_loc"], pk["xI"])]
        self.first.append(torch.tensor(rs.view(np.uint8), device=dev))
        self.now = [torch.empty_like(a) for a in self.first]
        self.off = torch.tensor(offs[:-1].astype(np.int64), device=dev)
        self.cap = torch.tensor(sizes.astype(np.int32), device=dev)

    def run(self):
        for d, s in zip(self.now, self.first):
            d.copy_(s)
        prim, x, dx, dtl, xI, rs = self.now
        gpu.step_tubes_noalloc(self.cfg, self.runs, self.total, self.off.data_ptr(), self.cap.data_ptr(),
                               rs.data_ptr(), prim.data_ptr(), x.data_ptr(), dx.data_ptr(), dtl.data_ptr(),
                               xI.data_ptr(), self.case["steps"],
                               stream=torch.cuda.current_stream().cuda_stream, stats=False)
        times = rs.view(torch.float64).view(self.runs, 4)[:, 1:3]  # t and dt of each run record
        return {"prim": prim, "x": x, "dx": dx, "dt_loc": dtl, "xI": xI, "t_dt": times}


def _pool_work(case):
    sizes = _sizes(case)
    zones = int(sizes[np.cumsum((sizes + 5) & ~1) <= 680000].sum()) * case["steps"]
    return {"bytes": 2. * 8 * 9 * zones, "flops": 550. * (1 if case["timestep"] == "euler" else 3) * zones}


# ---------------------------------------------------------------------------
# Blandford-McKee blast waves (1D spherical)


def _blast_setups(case, seed):
    """Seeded parameters as in the benchmark's sweep: E_iso, n and N log-spaced cells."""
    rng = np.random.default_rng(seed)
    return [problems.Bm1dSetup(eta=1e-10, lorentz_mode=1, lfac_shock2=1e4, Etot=10. ** float(rng.uniform(50., 54.)),
                               n_ext=10. ** float(rng.uniform(-3., 1.)), ncell=int(n), nmax=int(n) + 200, grid_log=1,
                               r_lo=.9, r_hi=1.1) for n in _sizes(case)]


def _blast_state(s):
    """The initial track of one run, whole arrays at a time."""
    d, n, g = s.derived(), s.ncell, s.ngst
    r_in, r_out = s.r_lo * d["RShock"] / d["lNorm"], s.r_hi * d["RShock"] / d["lNorm"]
    edge = r_in * np.exp(math.log(r_out / r_in) * np.arange(n + 1) / n)
    x, dx = np.zeros(n + 2 * g), np.zeros(n + 2 * g)
    x[g:-g], dx[g:-g] = .5 * (edge[:-1] + edge[1:]), edge[1:] - edge[:-1]
    r = x[g:-g] * d["lNorm"]
    ambient = r > d["RShock"]
    chi = np.where(ambient, 1., (1. + 2. * 4. * d["lfacShock2"]) * (1. - r / (problems.C_LIGHT * d["tstart"])))
    lfac = np.sqrt(d["lfacf"] ** 2 / chi + 1.)
    rho_a = s.n_ext * problems.MP
    prim = np.zeros((10, n + 2 * g))
    a = slice(g, n + g)
    prim[0, a] = np.where(ambient, rho_a, d["Df"] * chi ** (-7. / 4.) / lfac) / d["rhoNorm"]
    prim[1, a] = np.where(ambient, s.eta * rho_a * problems.C_LIGHT ** 2, d["pf"] * chi ** (-17. / 12.)) / d["pNorm"]
    prim[2, a] = np.where(ambient, 0., np.sqrt(lfac ** 2 - 1.))
    prim[4, a] = np.where(ambient, 1., 2.)
    prim[6, a] = prim[7, a] = np.cbrt(prim[0, a])
    xI = x[:-1] + dx[:-1] / 2.
    xI[g - 1] = x[g] - dx[g] / 2.
    problems._update_ghosts(prim, x, dx, xI, g)
    s._user_boundaries(prim, x, d["tstart"])
    return problems.TrackState(n + 2 * g, s.capacity, prim, x, dx, xI, np.full(n + 2 * g, problems.DT_INF),
                               d["tstart"], 0)


def _blast(case, seed):
    setups = _blast_setups(case, seed)
    states, params, cfg = [_blast_state(s) for s in setups], [s.run_params() for s in setups], gpu.config_sph()
    if case["settle"]:  # resume from the snapshot that a first job of a few steps left
        job = _Job1D(cfg, [s.capacity for s in setups], dict(case, tune=False), params)
        job.fill(states)
        job.g.step(case["settle"])
        got = job.g.download()
        states = [problems.unpack(got, r, job.g.offsets) for r in range(case["runs"])]
        job.g.close()
    job = _Job1D(cfg, [s.capacity for s in setups], case, params)
    job.fill(states)
    return job


def _blast_work(case):
    # a settled run keeps about a third of its log cells
    zones = int(_sizes(case).sum()) * case["steps"] * (.32 if case["settle"] else .6)
    return {"bytes": 2. * 8 * 13 * zones, "flops": 900. * 3 * zones}


# ---------------------------------------------------------------------------
# theta tracks (2D)


class _Jet:
    def __init__(self, case, seed):
        rng = np.random.default_rng(seed)
        s = problems.Jet2dSetup(ncell=case["ncell"], ntheta=case["ntheta"], nmax=case["ncell"] + case["ncell"] // 8 + 32,
                                Etot=10. ** float(rng.uniform(52.5, 53.5)), n_ext=10. ** float(rng.uniform(-.5, .5)),
                                th_max=.2, th_jet=float(rng.uniform(.08, .12)), merge_DR_slow=.3)
        self.steps = case["steps"]
        th, dth = s.theta()
        self.g = g = gpu2d.Grid2DGPU(s.ntheta, s.nmax, th, dth)
        g.set_params(s.params())
        g.upload(s.initial_state(), run_ghosts=True)
        g.step(case["settle"])
        # the snapshot a job resumes from, in pinned memory
        self.snap = st = g.download()
        for k in ("prim", "x", "dx", "xI", "dt_loc", "grad_mv", "grad_f1"):
            a = getattr(st, k)
            p = _pinned(*a.shape)
            p.numpy()[:] = a
            setattr(st, k, p.numpy())
        st.extra = {}
        NC = g.NC
        self.out = {"prim": _pinned(10, NC), "x": _pinned(1, NC), "dx": _pinned(1, NC), "xI": _pinned(1, NC)}
        self.nt = np.zeros(g.NJ, np.int32)

    def run(self):
        g, o = self.g, self.out
        g.upload(self.snap)
        g.step(self.steps)
        t, dt, it = ctypes.c_double(), ctypes.c_double(), ctypes.c_longlong()
        p = lambda a: ctypes.c_void_p(a.data_ptr())  # noqa: E731
        rc = gpu2d.lib().gamma_2d_download(g.h, ctypes.c_void_p(self.nt.ctypes.data), ctypes.byref(t),
                                           ctypes.byref(dt), ctypes.byref(it), None, p(o["prim"]), p(o["x"]),
                                           p(o["dx"]), None, p(o["xI"]), *([None] * 6))
        if rc != gpu.GAMMA_OK:
            raise gpu.GammaError(rc)
        offs = np.arange(g.NJ) * g.cap
        for k, v in o.items():
            _blank(v.numpy(), offs, [g.cap] * g.NJ, [g.cap] * g.NJ, self.nt - 1 if k == "xI" else self.nt)
        return {"ntrack": self.nt.copy(), "t": t.value, "dt": dt.value, **o}

    def __del__(self):
        self.g.close()


def _jet_work(case):
    zones = case["ntheta"] * case["ncell"] * case["steps"]
    # primitives, both gradients, geometry, dt_loc and lists read and written
    return {"bytes": 2. * (8 * 34 + 16) * zones, "flops": 2600. * 3 * zones}


# ---------------------------------------------------------------------------
# primitive recovery of independent states


def _c2p_inputs(case, seed):
    """States over the network's training range: lfac in [1, 1e3], p/rho in
    [1e-10, 1e3], rho in [1e-6, 1e6] (log-uniform), and their conserved variables."""
    rng = np.random.default_rng(seed)
    n, nq = case["n"], 10 if case["hydro"] == "sph" else 6
    lfac = np.exp(rng.uniform(0., math.log(1e3), n))
    rho = 10. ** rng.uniform(-6., 6., n)
    p = rho * 10. ** rng.uniform(-10., 3., n)
    u = np.sqrt(lfac * lfac - 1.) * rng.choice([-1., 1.], n)
    G = 4. / 3. if nq == 10 else 5. / 3.
    h = 1. + p * G / (G - 1.) / rho
    prim, cons = np.zeros((nq, n)), np.zeros((nq, n))
    D = lfac * rho
    cons[0], cons[1], cons[2], cons[4] = D, D * h * lfac - p - D, D * h * u, D
    prim[0], prim[1], prim[2], prim[4] = rho, p, u, 1.
    if case["start"] == "warm":  # the previous step's pressure
        prim[1] *= 1. + .02 * rng.uniform(-1., 1., n)
    else:
        prim[1] = 1.
    return prim, cons, G


def _network(seed, G):
    """A network for the starting pressure: fixed hidden layers, the output
    layer fitted to drawn states by least squares.  Parameters in the layout
    of gamma_mlp_init (W1 [64][3], b1, W2 [64][64], b2, W3 [2][64], b3)."""
    rng = np.random.default_rng(seed)
    m, H = 8000, 64
    lfac = np.exp(rng.uniform(0., math.log(1e3), m))
    rho = 10. ** rng.uniform(-6., 6., m)
    p = rho * 10. ** rng.uniform(-10., 3., m)
    D, h = lfac * rho, 1. + p * G / (G - 1.) / rho
    S, tau = D * h * np.sqrt(lfac * lfac - 1.), D * h * lfac - p - D
    f = np.stack([np.log1p(S / D) / 8., np.log10(np.maximum(tau / D - (np.sqrt(1. + (S / D) ** 2) - 1.), 1e-30)) / 10.,
                  np.log10(D) / 6.], 1)
    silu = lambda z: z / (1. + np.exp(-z))  # noqa: E731
    W1, b1 = rng.normal(0., 1.5, (H, 3)), rng.uniform(-1., 1., H)
    W2, b2 = rng.normal(0., .3, (H, H)), rng.uniform(-.5, .5, H)
    a = silu(silu(f @ W1.T + b1) @ W2.T + b2)
    A = np.concatenate([a, np.ones((m, 1))], 1)
    y = np.stack([(np.log(p / D) + 14.) / 10., np.log(lfac) / 3.], 1)
    X = np.linalg.solve(A.T @ A + 1e-3 * np.eye(H + 1), A.T @ y)
    return np.concatenate([W1.ravel(), b1, W2.ravel(), b2, X[:H].T.ravel(), X[H]]).astype(np.float32)


class _C2P:
    def __init__(self, case, seed):
        prim, cons, G = _c2p_inputs(case, seed)
        dev = torch.device("cuda")
        self.case, self.cfg = case, gpu.config_sph() if case["hydro"] == "sph" else gpu.config_cart()
        self.prim0, self.cons0 = torch.tensor(prim, device=dev), torch.tensor(cons, device=dev)
        self.prim, self.cons = torch.empty_like(self.prim0), torch.empty_like(self.cons0)
        self.P = torch.tensor(_network(seed, G), device=dev) if case["start"] == "learned" else None

    def run(self):
        self.prim.copy_(self.prim0)
        self.cons.copy_(self.cons0)
        s, n = torch.cuda.current_stream().cuda_stream, self.case["n"]
        if self.P is None:
            gpu.cons2prim_device(self.cfg, self.cons.data_ptr(), self.prim.data_ptr(), n, stream=s)
        else:
            gpu.cons2prim_guess_device(self.cfg, self.cons.data_ptr(), self.prim.data_ptr(), n, self.P.data_ptr(),
                                       stream=s)
        return {"prim": self.prim, "cons": self.cons}


def _c2p_work(case):
    nq = 10 if case["hydro"] == "sph" else 6
    its = {"cold": 12., "warm": 3., "learned": 4.}[case["start"]]
    return {"bytes": 8. * nq * 4 * case["n"], "flops": (30. * its + 60.) * case["n"]}


def _c2p_exact(case, seed):
    prim, cons, G = _c2p_inputs(case, seed)
    parts = [_recover(*(a[k:k + 32768] for a in cons[:3]), G, prim[1, k:k + 32768])  # a block that fits the cache
             for k in range(0, case["n"], 32768)]
    p, rho, u = (np.concatenate(a) for a in zip(*parts))
    p = np.maximum(p, 1e-10 if case["hydro"] == "sph" else 0.)
    out = np.zeros_like(prim)
    out[0], out[1], out[2] = rho, p, u
    out[4:] = cons[4:] / cons[0]
    lf = np.sqrt(1. + u * u)
    h, D = 1. + p * G / (G - 1.) / rho, lf * rho
    c = np.zeros_like(cons)
    c[0], c[1], c[2] = D, D * h * lf - p - D, D * h * u
    c[4:] = out[4:] * D
    return {"prim": out, "cons": c}


def _recover(D, tau, S, G, start):
    """p, rho, u of conserved states: Newton inside a bracket on
    E + p - D lfac - p lfac^2 G / (G - 1) = 0."""
    E, k = D + tau, G / (G - 1.)
    aS = np.abs(S)

    def f(p):
        W = E + p
        v2 = (S / W) ** 2
        l2 = 1. / np.abs(1. - v2)
        l = np.sqrt(l2)
        dl = -l * l2 * v2 / W
        return W - D * l - k * p * l2, 1. - D * dl - k * (l2 + 2. * p * l * dl)
    lo = np.maximum(0., (1. + 1e-13) * aS - E)
    p = np.maximum(start, lo * (1. + 1e-12) + 1e-300)
    hi = p.copy()
    for _ in range(400):
        up = f(hi)[0] > 0.
        if not up.any():
            break
        hi = np.where(up, hi * 10., hi)
    p = np.clip(start, lo, hi)
    for _ in range(60):
        v, d = f(p)
        lo, hi = np.where(v > 0., p, lo), np.where(v < 0., p, hi)
        q = p - v / d
        mid = np.where(lo > 0., np.sqrt(lo) * np.sqrt(hi), .5 * (lo + hi))
        q = np.where((q > lo) & (q < hi), q, mid)
        q = np.where(v == 0., p, q)
        if np.all(np.abs(q - p) <= 1e-15 * p):
            break
        p = q
    W = E + p
    w = np.sqrt(np.maximum((W - aS) * (W + aS), 0.))  # W / lfac
    return p, D * w / W, S / w


# ---------------------------------------------------------------------------
# training


def _train_inputs(case, seed):
    rng = np.random.default_rng(seed)
    n, H = case["n"], 64
    lfac = np.exp(rng.uniform(0., math.log(1e3), n))
    rho = 10. ** rng.uniform(-6., 6., n)
    p = rho * 10. ** rng.uniform(-10., 3., n)
    D, h = lfac * rho, 1. + 4. * p / rho
    s, th = h * np.sqrt(lfac * lfac - 1.), h * lfac - p / D - 1.
    x = np.stack([np.log1p(s) / 8., np.log10(np.maximum(th - (np.sqrt(1. + s * s) - 1.), 1e-30)) / 10.,
                  np.log10(D) / 6.], 1).astype(np.float32)
    y = np.stack([(np.log(p / D) + 14.) / 10., np.log(lfac) / 3.], 1).astype(np.float32)
    P = np.concatenate([rng.uniform(-1., 1., 3 * H) * math.sqrt(6. / (3 + H)), np.zeros(H),
                        rng.uniform(-1., 1., H * H) * math.sqrt(6. / (2 * H)), np.zeros(H),
                        rng.uniform(-1., 1., 2 * H) * math.sqrt(6. / (H + 2)), np.zeros(2)]).astype(np.float32)
    return x, y, P


class _Train:
    def __init__(self, case, seed):
        dev = torch.device("cuda")
        self.case = case
        self.x, self.y, self.P0 = (torch.tensor(a, device=dev) for a in _train_inputs(case, seed))
        self.P = torch.empty_like(self.P0)

    def run(self):
        self.P.copy_(self.P0)
        c = self.case
        loss = gpu.mlp_train(self.P.data_ptr(), self.x.data_ptr(), self.y.data_ptr(), c["n"], epochs=c["epochs"],
                             batch=c["batch"], stream=torch.cuda.current_stream().cuda_stream)
        return {"params": self.P, "loss": loss}


def _train_work(case):
    return {"bytes": 20. * case["n"] * case["epochs"], "flops": 6. * 4546 * case["n"] * case["epochs"]}


# ---------------------------------------------------------------------------
# planar tubes in 64 bits, plain numpy: one tube after another


def _minmod(a, b):
    out = np.where((np.abs(a) < np.abs(b)) & (a * b > 0.), a, 0.)
    return np.where((np.abs(b) < np.abs(a)) & (a * b > 0.), b, out)


def _fluxes(q, xI, cen, G):
    """HLLC at interfaces that move with the contact: fluxes, speeds."""
    g = (q[:, 1:] - q[:, :-1]) / (cen[1:] - cen[:-1])
    L, R = q[:, :-1].copy(), q[:, 1:].copy()
    m = _minmod(g[:, :-1], g[:, 1:])  # of cells 1 .. n-2
    L[:, 1:-1] += m[:, :-1] * (xI[1:-1] - cen[1:-2])
    R[:, 1:-1] += m[:, 1:] * (xI[1:-1] - cen[2:-1])
    out = []
    for s in (L, R):
        rho, p, u = s[:3]
        lf = np.sqrt(1. + u * u)
        D, h = lf * rho, 1. + p * G / (G - 1.) / rho
        v, m1 = u / lf, D * h * u
        cons = np.concatenate([np.stack([D, D * h * lf - p - D, m1]), s[3:] * D])
        flux = np.concatenate([np.stack([D * v, m1 - D * v, m1 * v + p]), s[3:] * D * v])
        cs2 = G * p / (rho + p * G / (G - 1.))
        sg = cs2 / (lf * lf * (1. - cs2))
        root = np.sqrt(sg * (1. - v * v + sg))
        out.append((cons, flux, v, p, (v - root) / (1. + sg), (v + root) / (1. + sg)))
    (cL, fL, vL, pL, aL, bL), (cR, fR, vR, pR, aR, bR) = out
    lL, lR = np.minimum(aL, aR), np.maximum(bL, bR)
    EL, ER = cL[0] + cL[1], cR[0] + cR[1]
    AL, AR = lL * EL - cL[2], lR * ER - cR[2]
    BL, BR = cL[2] * (lL - vL) - pL, cR[2] * (lR - vR) - pR
    FE, Eh = (lL * AR - lR * AL) / (lR - lL), (AR - AL) / (lR - lL)
    Fm, mh = (lL * BR - lR * BL) / (lR - lL), (BR - BL) / (lR - lL)
    e = Eh + Fm
    flat = np.abs(FE) < 1e-15
    with np.errstate(all="ignore"):
        lS = np.where(flat, mh / e, (e - np.sqrt(e * e - 4. * FE * mh)) / (2. * np.where(flat, 1., FE)))
    v = lS
    fl = np.where(v < lL, fL - v * cL, 0.)
    for c, f, vv, p, lb, on in ((cL, fL, vL, pL, lL, (lL <= v) & (v < lS)), (cR, fR, vR, pR, lR, (lS <= v) & (v < lR))):
        E, m1 = c[0] + c[1], c[2]
        with np.errstate(all="ignore"):
            pS = ((lb * E - m1) * lS - (m1 * (lb - vv) - p)) / (1. - lb * lS)
            k = (lb - vv) / (lb - lS)
            sc = c * k
            sc[2] = (m1 * (lb - vv) + pS - p) / (lb - lS)
            sc[1] = (E * (lb - vv) + pS * lS - p * vv) / (lb - lS) - sc[0]
        fl = np.where(on, f + lb * (sc - c) - v * sc, fl)
    return np.where(lR <= v, fR - v * cR, fl), v, lL, lR


def _tube_exact(s, steps, G, cyl, euler):
    """Steps of one tube (cells outside the active ones are copies of the edge
    cells, moved outwards), after the SSP-RK3 and Euler time steps."""
    ng, n = 2, s.ntrack
    q = np.delete(s.prim, 3, 0)
    x, dx, dtl = s.x.copy(), s.dx.copy(), s.dt_loc.copy()
    xI = s.xI.copy()
    iL, iR = ng - 1, n - ng
    act = slice(iL + 1, iR)

    def ghosts():
        for i in range(iL + 1):
            q[:, i], dtl[i], dx[i] = q[:, iL + 1], dtl[iL + 1], dx[iL + 1]
            x[i] = x[iL + 1] - (iL - i + 1) * dx[iL + 1]
        for i in range(iR, n):
            q[:, i], dtl[i], dx[i] = q[:, iR - 1], dtl[iR - 1], dx[iR - 1]
            x[i] = x[iR - 1] + (i - iR + 1) * dx[iR - 1]
        for i in range(iL):
            xI[i] = xI[iL + 1] - (iL - i + 1) * dx[iL + 1]
        for i in range(iR, n - 1):
            xI[i] = xI[iR - 1] + (i - iR) * dx[iR - 1]

    def conserved(q):
        lf = np.sqrt(1. + q[2] ** 2)
        D, h = lf * q[0], 1. + q[1] * G / (G - 1.) / q[0]
        return np.concatenate([np.stack([D, D * h * lf - q[1] - D, D * h * q[2]]), q[3:] * D])

    def primitive(c, p0):
        p, rho, u = _recover(c[0], c[1], c[2], G, p0)
        return np.concatenate([np.stack([rho, p, u]), c[3:] / c[0]])

    for _ in range(steps):
        for stage in (1,) if euler else (1, 2, 3):
            ghosts()
            fl, v, lL, lR = _fluxes(q, xI, x, G)
            with np.errstate(divide="ignore", invalid="ignore"):
                a = dx[1:-1]
                cL = np.where(lR[:-1] > v[1:], a / (lR[:-1] - v[1:]), problems.DT_INF)
                cR = np.where(lL[1:] < v[:-1], a / (v[:-1] - lL[1:]), problems.DT_INF)
            dtl[1:-1] = np.minimum(dtl[1:-1], np.minimum(cL, cR))
            if stage == 1:
                dt = .2 * dtl.min()
                dtl[:] = problems.DT_INF
                xI0, u0 = xI.copy(), conserved(q)[:, act] * dx[act]
            c = conserved(q)[:, act] * dx[act] + (fl[:, iL:iR - 1] - fl[:, iL + 1:iR]) * dt
            if cyl:
                c[2] += q[1, act] / x[act] * dx[act] * dt
            xn = xI + dt * v
            dn = xn[iL + 1:iR] - xn[iL:iR - 1]
            new = primitive(c / dn, q[1, act])
            if stage > 1:
                w0, w1 = (.75, .25) if stage == 2 else (1. / 3., 2. / 3.)
                c = w0 * u0 + w1 * conserved(new) * dn
                xn[iL:iR] = w0 * xI0[iL:iR] + w1 * xn[iL:iR]
                dn = xn[iL + 1:iR] - xn[iL:iR - 1]
                new = primitive(c / dn, new[1])
            q[:, act] = new
            xI = xn
            inner = act if euler else slice(1, n - 1)
            if stage == (1 if euler else 3):
                lo, hi = inner.start, inner.stop
            else:
                lo, hi = act.start, act.stop
            x[lo:hi], dx[lo:hi] = (xI[lo:hi] + xI[lo - 1:hi - 1]) / 2., xI[lo:hi] - xI[lo - 1:hi - 1]
    return np.insert(q, 3, 0., 0), x, dx, dtl, xI


def _tubes_exact(case, seed):
    sizes = _sizes(case)
    euler, cyl = case["timestep"] == "euler", case["hydro"] == "cyl"
    if int(sizes.sum()) * case["steps"] > 200000 or case["runs"] * case["steps"] > 1000:
        return None  # minutes in numpy
    states = _tube_states(case, seed, sizes)
    nt = np.array([s.ntrack for s in states], np.int32)
    offs = np.concatenate([[0], np.cumsum((nt + 1) & ~1)])
    out = {k: np.zeros((6 if k == "prim" else 1, int(offs[-1]))) for k in ("prim", "x", "dx", "dt_loc", "xI")}
    for s, o in zip(states, offs):
        got = _tube_exact(s, case["steps"], 5. / 3., cyl, euler)
        for k, a in zip(("prim", "x", "dx", "dt_loc", "xI"), got):
            out[k][:, o:o + a.shape[-1]] = a
    return {"ntrack": None, **out}


def _train_exact(case, seed):
    """The same mini-batches (the sample order of gamma_mlp_train) and Adam in 64 bits."""
    x, y, P = _train_inputs(case, seed)
    n, H, M64 = case["n"], 64, (1 << 64) - 1
    if case["n"] * case["epochs"] > 1100000:
        return None
    P, m, w = P.astype(np.float64), np.zeros(P.size), np.zeros(P.size)
    cut = np.cumsum([0, 3 * H, H, H * H, H, 2 * H, 2])
    per = -(-n // case["batch"])
    total, step, losses = per * case["epochs"], 0, []

    def mix(z):
        z = (z + 0x9e3779b97f4a7c15) & M64
        z = ((z ^ (z >> 30)) * 0xbf58476d1ce4e5b9) & M64
        z = ((z ^ (z >> 27)) * 0x94d049bb133111eb) & M64
        return z ^ (z >> 31)
    muls = [1000003, 999983, 999979, 999961, 999959, 999953, 999931, 999917]
    for e in range(case["epochs"]):
        h = mix(7 ^ (0x1234567 + e))
        mul = next((c for c in (muls[(h + j) % 8] % n for j in range(8)) if c > 0 and math.gcd(c, n) == 1), 1)
        order = (mul * np.arange(n) + h % n) % n
        loss = 0.
        for b in range(per):
            k = order[b * case["batch"]:(b + 1) * case["batch"]]
            X, Y = x[k].astype(np.float64), y[k].astype(np.float64)
            W1, b1, W2, b2, W3, b3 = (P[i:j] for i, j in zip(cut[:-1], cut[1:]))
            W1, W2, W3 = W1.reshape(H, 3), W2.reshape(H, H), W3.reshape(2, H)
            z1 = X @ W1.T + b1
            s1 = 1. / (1. + np.exp(-z1))
            z2 = (z1 * s1) @ W2.T + b2
            s2 = 1. / (1. + np.exp(-z2))
            r = (z2 * s2) @ W3.T + b3 - Y
            loss += .5 * float((r * r).sum()) / len(k)
            d3 = r / len(k)
            d2 = (d3 @ W3) * (s2 + z2 * s2 * (1. - s2))
            d1 = (d2 @ W2) * (s1 + z1 * s1 * (1. - s1))
            grad = np.concatenate([(d1.T @ X).ravel(), d1.sum(0), (d2.T @ (z1 * s1)).ravel(), d2.sum(0),
                                   (d3.T @ (z2 * s2)).ravel(), d3.sum(0)])
            frac = step / (total - 1) if total > 1 else 0.
            lr = 1e-4 + .5 * (3e-3 - 1e-4) * (1. + math.cos(math.pi * frac))
            step += 1
            m, w = .9 * m + .1 * grad, .999 * w + .001 * grad * grad
            P = P - lr * (m / (1. - .9 ** step)) / (np.sqrt(w / (1. - .999 ** step)) + 1e-8)
        losses.append(loss / per)
    return {"params": P, "loss": np.array(losses)}


# prepare, work, exact of each kind.  The blast waves and the jets have no
# exact values here: their regrid decides on the live track, cell by cell, and
# their limiter and neighbour order are the reference's own.  The tubes in the
# caller's arrays are those of "tubes".
_KINDS = {
    "tubes": (_tubes, _tubes_work, _tubes_exact),
    "pool": (_Pool, _pool_work, None),
    "blast": (_blast, _blast_work, None),
    "jet": (_Jet, _jet_work, None),
    "c2p": (_C2P, _c2p_work, _c2p_exact),
    "train": (_Train, _train_work, _train_exact),
}
