"""The workloads whose speed is tracked: what programs have this framework do,
from the smallest scene to the largest, through the public entry points.

A simulation case is one run as the ``sphere`` executable makes it between
reading an input file and writing an output file: upload of the particle
state from pinned host memory, ``steps`` time steps, download of the output
file's fields.  The other kinds are an ensemble of scenes in one context, one
iteration of a calibration loop (forward and adjoint), a run with the Darcy
flow, one ray-traced frame, and the cell list of positions that are on the
device already.

``exact`` restates the paths in plain torch at 64 bits.  Lengths are narrowed
to a float square root there, as the force laws define them; the
differentiable step is defined with exact lengths.
"""
import ctypes as C
import math

import numpy as np
import torch
from torch.utils.checkpoint import checkpoint

from sphere_b200 import scenes, sphk
from sphere_b200.darcy import DarcyState
from sphere_b200.spherebin import Spherebin
from sphere_b200.state import config_from_spherebin, state_from_spherebin

# what an output file holds of the particles, the walls and the bonds
FIELDS = ("x", "xysum", "vel", "force", "angpos", "angvel", "torque", "es_dot", "es", "ev_dot",
          "ev", "p", "walls_nx", "walls_mvfd", "bonds", "bonds_delta", "bonds_omega")
FLOW_FIELDS = ("H", "V", "K", "phi", "dphi")
NU = 8.9e-4            # viscosity of water, Pa s


def listed():
    return [
        # a test scene in the open: every kernel is short, so launches and latency count
        dict(name="collision_500", kind="collision", n=500, nw=0, model=2, steps=200),
        # the settling scene that the benchmark runs on the CPU too: 10,000 grains falling freely
        dict(name="settling_10k", kind="settling", nx=20, ny=20, nz=25, steps=500),
        # a rapid flow: contacts open, close and slide, and grains change cells, in every step
        dict(name="collision_50k", kind="collision", n=50021, nw=1, model=2, steps=200),
        # the same with linear-viscous contacts and capillary bridges
        dict(name="cohesive_20k", kind="collision", n=20011, nw=1, model=1, steps=100),
        # the benchmark's 1M grains: polydisperse, hardly in contact, under a loaded wall
        dict(name="loose_1m", kind="loose", n=1000000, steps=1000),
        # the benchmark's jammed column: six contacts a grain
        dict(name="packed_1m", kind="packed", nx=100, ny=100, nz=100, steps=500),
        # the benchmark's bonded bar at a quarter of its size, until its bonds fail
        dict(name="bonded_75k", kind="bonded", nx=37, ny=23, nz=22, steps=500),
        # a parameter study: scenes of 500 to 20,000 grains, in contact from the start
        dict(name="ensemble_64", kind="ensemble", members=64, jammed=True, steps=300),
        # calibration on the benchmark's jammed column, with a shorter run
        dict(name="adjoint_100k", kind="adjoint", nx=40, ny=40, nz=63, steps=200, every=50),
        # pore water in a bed
        dict(name="darcy_250k", kind="darcy", n=250000, steps=100),
        # one frame of a movie of the 1M grains
        dict(name="render_1m", kind="render", n=1000000, width=800, height=800, method=2),
        # neighbour search of a caller's own positions
        dict(name="cells_1m", kind="cells", n=1000000, num_x=50, num_y=50, num_z=100),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("collision", "settling", "cohesive", "loose", "packed", "bonded", "ensemble",
                       "adjoint", "darcy", "render", "cells"))
    if kind in ("collision", "cohesive"):
        return dict(kind="collision", n=_log(rng, 200, 100000), nw=rng.randint(0, 1),
                    model=2 if kind == "collision" else 1, steps=rng.randint(40, 200))
    if kind == "settling":
        return dict(kind=kind, nx=rng.randint(5, 20), ny=rng.randint(5, 20), nz=rng.randint(3, 50),
                    steps=rng.randint(100, 500))
    if kind == "loose":
        return dict(kind=kind, n=_log(rng, 20000, 1000000), steps=rng.randint(200, 900))
    if kind == "packed":
        n = _log(rng, 5000, 1000000)
        nx, ny = (max(6, int(n ** (1 / 3) * rng.uniform(0.7, 1.4))) for _ in range(2))
        return dict(kind=kind, nx=nx, ny=ny, nz=max(2, n // (nx * ny)), steps=rng.randint(100, 450))
    if kind == "bonded":
        return dict(kind=kind, nx=rng.randint(8, 40), ny=rng.randint(4, 23), nz=rng.randint(4, 23),
                    steps=rng.randint(100, 500))
    if kind == "ensemble":
        return dict(kind=kind, members=rng.randint(3, 64), jammed=rng.random() < 0.5,
                    steps=rng.randint(100, 300))
    if kind == "adjoint":
        return dict(kind=kind, nx=rng.randint(8, 40), ny=rng.randint(8, 40), nz=rng.randint(8, 60),
                    steps=rng.randint(60, 200), every=rng.randint(20, 60))
    if kind == "darcy":
        return dict(kind=kind, n=_log(rng, 10000, 300000), steps=rng.randint(40, 100))
    if kind == "render":
        return dict(kind=kind, n=_log(rng, 1000, 1000000), width=rng.randint(100, 1000),
                    height=rng.randint(100, 1000), method=rng.randint(0, 5))
    num = [rng.randint(5, 80) for _ in range(3)]
    return dict(kind=kind, n=_log(rng, 500, 1000000), num_x=num[0], num_y=num[1], num_z=num[2])


# ---- scenes -----------------------------------------------------------------

def _loose(n, seed):
    """n grains of the benchmark's log-normal radii, each inside its own site
    of a cubic lattice and so clear of its neighbours, in random motion, with
    periodic sides and a loaded top wall."""
    rng = np.random.default_rng(seed)
    s = 2.52e-3
    m = max(3, int(round(n ** (1.0 / 3.0))))
    i = np.arange(n)
    sb = Spherebin(np_=n, nw=1)
    sb.radius = np.clip(np.exp(rng.normal(math.log(1e-3), 0.2, n)), 0.5e-3, 1.25e-3)
    sb.x = (np.stack([i % m, (i // m) % m, i // (m * m)], axis=1) + 0.5) * s
    sb.x += rng.uniform(-1.0, 1.0, (n, 3)) * (0.5 * s - sb.radius)[:, None]
    sb.vel = rng.uniform(-0.05, 0.05, (n, 3))
    sb.angvel = rng.uniform(-20.0, 20.0, (n, 3))
    sb.L = np.array([m * s, m * s, -(-n // (m * m)) * s + 8e-3])
    sb.num = np.maximum(3, np.floor(sb.L / 4e-3)).astype(np.uint32)
    sb.periodic = 1
    sb.g = np.array([0.0, 0.0, -9.81])
    sb.k_n = sb.k_t = 1e6
    sb.gamma_n, sb.gamma_wn, sb.gamma_wt = 0.01, 3.0, 3.0
    sb.mu_s = sb.mu_d = sb.mu_ws = sb.mu_wd = 0.5
    sb.wmode = np.array([1], dtype=np.int32)
    sb.w_x = np.array([float(np.max(sb.x[:, 2] + sb.radius))])
    sb.w_m = np.array([sb.rho * n * math.pi * 2e-3 ** 3])
    sb.w_devs = np.array([20e3])
    sb.time_dt = 2e-7
    return sb


def _scenes(case, seed):
    kind = case["kind"]
    if kind == "collision":
        side = (case["n"] * 8.2e-9 / 0.35) ** (1.0 / 3.0)
        sb = scenes.collision(n=case["n"], seed=seed, nw=case["nw"], box=(1.2 * side + 0.012,) * 3,
                              phi_target=0.35, k_n=500.0, k_t=500.0, gamma_n=0.01)
        if case["model"] == 1:
            sb.contactmodel, sb.kappa, sb.V_b, sb.db = 1, 0.05, 1e-12, 1e-4
        return [sb]
    if kind == "settling":
        return [scenes.settling(seed, case["nx"], case["ny"], case["nz"])]
    if kind == "packed":
        return [scenes.packed(case["nx"], case["ny"], case["nz"], seed=seed,
                              height=4e-3 * (case["nz"] // 2 + 3))]
    if kind == "bonded":
        return [scenes.tension(case["nx"], case["ny"], case["nz"], seed=seed)]
    if kind == "adjoint":
        return [scenes.jammed_column(case["nx"], case["ny"], case["nz"], seed=seed)]
    if kind == "ensemble":
        make = scenes.jammed_member if case["jammed"] else scenes.ensemble_member
        k = case["members"]
        sizes = [int(round(500.0 * 40.0 ** ((j + 0.5) / k))) for j in range(k)]
        return [make(64 * (seed % 1000000) + j, n_range=(n, n)) for j, n in enumerate(sizes)]
    return [_loose(case["n"], seed)]


def _pinned(st):
    """The file's fields of a host state in pinned memory; the rest (contact
    slots, half-step velocities) stays on the device, as in a plain run."""
    for name, v in list(st.__dict__.items()):
        if isinstance(v, np.ndarray):
            setattr(st, name, _pin(v) if name in FIELDS and v.size else
                    v if name in FIELDS else None)
    return st


def _pin(a):
    t = torch.empty(a.shape, dtype=torch.from_numpy(a.reshape(-1)[:0]).dtype, pin_memory=True)
    t.numpy()[...] = a
    return t.numpy()


def _pressure(cfg, seed):
    """A fluid grid with an uneven starting pressure, set up as the reference does."""
    ds = DarcyState.zeros(cfg.num)
    rng = np.random.default_rng(seed + 1)
    ds.set_cells(H=rng.uniform(0.9e4, 1.1e4, tuple(int(v) for v in cfg.num)))
    return ds


class _State:
    pass


def prepare(case, seed):
    s = _State()
    s.case = case
    if case["kind"] == "cells":
        gen = torch.Generator(device="cuda").manual_seed(seed)
        n, num = case["n"], [case["num_x"], case["num_y"], case["num_z"]]
        s.x = torch.rand((n, 4), generator=gen, device="cuda", dtype=torch.float64)
        s.x *= torch.tensor([4e-3 * v for v in num] + [1e-3], device="cuda", dtype=torch.float64)
        sb = Spherebin(np_=1, nw=0)
        sb.L, sb.num, sb.time_dt = np.array([4e-3 * v for v in num]), np.array(num), 1.0
        s.conf = sphk.make_config(config_from_spherebin(sb))
        s.conf.np = n
        s.out = [torch.empty(k, dtype=torch.int32, device="cuda") for k in (n, n, math.prod(num), math.prod(num))]
        s.lib = sphk.load_library()
        return s
    sbs = _scenes(case, seed)
    cfgs = [config_from_spherebin(sb) for sb in sbs]
    states = [state_from_spherebin(sb) for sb in sbs]
    if case["kind"] == "ensemble":
        s.sim = sphk.BatchSimulation(cfgs)
        st = sphk.pack_states(states)
    else:
        s.sim = sphk.Simulation(cfgs[0])
        st = states[0]
    s.state = _pinned(st)
    s.result = _pinned(st.copy())
    if case["kind"] == "render":
        s.sim.upload(s.state)
        s.sim.step(1)
        s.sim.sync()
    elif case["kind"] == "darcy":
        s.sim.upload(s.state)
        ds = _pressure(cfgs[0], seed)
        sphk.darcy_init(cfgs[0], NU, st.x, ds)
        s.sim.darcy_upload(ds, NU)
        s.flow = ds
        for name, v in ds.arrays().items():
            setattr(s.flow, name, _pin(v))
    elif case["kind"] == "adjoint":
        s.x_bar, s.v_bar = _seeds(case, seed)
    return s


def _seeds(case, seed):
    """Derivatives of a loss with respect to the final positions and velocities."""
    rng = np.random.default_rng(seed + 2)
    n = case["nx"] * case["ny"] * case["nz"]
    return rng.normal(0.0, 1.0, (n, 3)), rng.normal(0.0, 1e-3, (n, 3))


def run(s):
    case, kind = s.case, s.case["kind"]
    if kind == "cells":
        stream = torch.cuda.current_stream().cuda_stream
        rc = s.lib.sph_cell_list_noalloc(C.byref(s.conf), C.c_void_p(s.x.data_ptr()),
                                         *(C.c_void_p(o.data_ptr()) for o in s.out),
                                         C.c_void_p(stream))
        if rc != 0:
            raise sphk.SphError(rc, "cell list")
        return s.out
    if kind == "render":
        return s.sim.render(case["method"], 0.05, 0.0, case["width"], case["height"])
    sphk.Simulation.upload(s.sim, s.state)   # an ensemble's packed state too
    if kind == "adjoint":
        s.sim.diff_begin(checkpoint_every=case["every"])
        s.sim.step(case["steps"])
        s.sim.sync()
        s.sim.download(s.result)
        g = s.sim.diff_backward(s.x_bar, s.v_bar)
        s.sim.diff_end()
        return {"x": s.result.x, "vel": s.result.vel, "k_n": g["k_n"], "k_t": g["k_t"],
                "gamma_n": g["gamma_n"], "mu": g["mu"], "x0": g["x0"], "v0": g["v0"]}
    s.sim.step(case["steps"])
    s.sim.sync()
    s.sim.download(s.result)
    out = {f: getattr(s.result, f) for f in FIELDS if getattr(s.result, f).size}
    if kind == "darcy":
        s.sim.darcy_download(s.flow)
        out.update({f: getattr(s.flow, f) for f in FLOW_FIELDS})
    return out


def work(case):
    """Bytes of one pass: a particle's state read and written once a step (192
    + 176), its cell-list entry (16), each cell's bounds (16), each directed
    contact's slot (52) and each bond's history (136); the adjoint runs every
    step three times (forward, recorded, reversed)."""
    kind = case["kind"]
    if kind == "cells":
        return {"bytes": 40.0 * case["n"] + 8.0 * case["num_x"] * case["num_y"] * case["num_z"]}
    if kind == "render":
        return {"bytes": 60.0 * case["n"] + 4.0 * case["width"] * case["height"]}
    contacts = bonds = flow = 0
    if "nx" in case:
        n = case["nx"] * case["ny"] * case["nz"]
        cells = n / 4
        if kind in ("packed", "adjoint"):
            contacts = 6 * n
        if kind == "bonded":
            n, bonds, cells = 4 * n, 23 * n, 4 * n
        if kind == "settling":
            cells = 24 * 24 * 96
    elif kind == "ensemble":
        k = case["members"]
        n = sum(500.0 * 40.0 ** ((j + 0.5) / k) for j in range(k))
        contacts, cells = (6 * n if case["jammed"] else 0), n / 2
    else:
        n = case["n"]
        contacts, cells = (2 * n if kind == "collision" else 0), n / 2
        if kind == "darcy":
            cells = n / 4
            flow = 4 * n + 248 * cells
    step = 384.0 * n + 16.0 * cells + 52.0 * contacts + 136.0 * bonds + flow
    return {"bytes": step * case["steps"] * (3 if kind == "adjoint" else 1)}


def tolerance(case):
    # Everything is the reference's arithmetic in its own order, bit for bit,
    # but the adjoint, whose sums over contacts have no fixed order.  The same
    # inputs twice differ by 1e-14; the derivative with respect to k_n, a sum
    # that cancels, is 1.5e-8 off the 64-bit restatement, where the rounding
    # of each contact differs: four times that.
    return {"rel": 6e-8, "max": 2.4e-6} if case["kind"] == "adjoint" else "exact"


# ---- the paths at 64 bits -----------------------------------------------------

def exact(case, seed):
    kind = case["kind"]
    if kind in ("cells", "render"):
        return None   # whole numbers
    sbs = _scenes(case, seed)
    bed = _Bed(sbs, case["steps"], smooth=kind == "adjoint")
    if bed.cost * case["steps"] * (4 if kind == "adjoint" else 1) > 6e9:
        return None
    if kind == "adjoint":
        return _exact_adjoint(bed, case, seed)
    flow = _Flow(bed, _pressure(config_from_spherebin(sbs[0]), seed)) if kind == "darcy" else None
    st = bed.start()
    for _ in range(case["steps"]):
        if flow is not None:
            flow.step(st["x"])
        st = bed.step(st)
    out = bed.fields(st)
    if flow is not None:
        out.update(flow.fields())
    return out


def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _t(a):
    return torch.as_tensor(np.ascontiguousarray(a, dtype=np.float64), device=_dev())


def _dot(a, b):
    return a[:, 0:1] * b[:, 0:1] + a[:, 1:2] * b[:, 1:2] + a[:, 2:3] * b[:, 2:3]


def _cross(a, b):
    return torch.linalg.cross(a, b, dim=1)


def _pairs(xa, ra, xb, rb, L, periodic, margin, same):
    """Every (a, b) with |xa - xb| < ra + rb + margin, through the nearest
    image on periodic axes; without a = b when `same`."""
    reach = float(ra.max() + rb.max()) + margin
    num = [max(1, int(v / reach)) for v in L]
    size = _t([v / k for v, k in zip(L, num)])
    top = torch.tensor(num, device=xa.device) - 1

    def cell(x):
        return torch.minimum(torch.floor(x / size).long().clamp(min=0), top)

    def key(c):
        return c[:, 0] + num[0] * (c[:, 1] + num[1] * c[:, 2])

    kb, order = torch.sort(key(cell(xb)))
    ca = cell(xa)
    seen, got_a, got_b = set(), [], []
    for o in range(27):
        off = [o % 3 - 1, o // 3 % 3 - 1, o // 9 - 1]
        fold = tuple(v % num[q] if periodic[q] else v for q, v in enumerate(off))
        if fold in seen:
            continue
        seen.add(fold)
        c, ok = ca.clone(), torch.ones(len(ca), dtype=torch.bool, device=xa.device)
        for q in range(3):
            c[:, q] += off[q]
            if periodic[q]:
                c[:, q] %= num[q]
            else:
                ok &= (c[:, q] >= 0) & (c[:, q] < num[q])
        a = torch.nonzero(ok)[:, 0]
        k = key(c[a])
        lo = torch.searchsorted(kb, k)
        cnt = torch.searchsorted(kb, k, right=True) - lo
        a2 = torch.repeat_interleave(a, cnt)
        first = torch.repeat_interleave(lo - (torch.cumsum(cnt, 0) - cnt), cnt)
        b = order[first + torch.arange(len(a2), device=xa.device)]
        d = xa[a2] - xb[b]
        for q in range(3):
            if periodic[q]:
                d[:, q] -= L[q] * torch.round(d[:, q] / L[q])
        near = _dot(d, d)[:, 0] < (ra[a2, 0] + rb[b, 0] + margin) ** 2
        if same:
            near &= a2 != b
        got_a.append(a2[near])
        got_b.append(b[near])
    return torch.cat(got_a), torch.cat(got_b)


class _Bed:
    """The grains of one or several scenes and the law of their motion."""

    NAMES = ("k_n", "k_t", "gamma_n", "gamma_t", "mu_s", "mu_d", "gamma_wn", "gamma_wt", "mu_ws",
             "mu_wd", "rho", "kappa", "db", "V_b")

    def __init__(self, sbs, steps, smooth=False):
        self.sbs, self.sb, self.smooth = sbs, sbs[0], smooth
        per = lambda f: _t(np.concatenate([np.broadcast_to(f(sb), (sb.np, np.size(f(sb))))  # noqa: E731
                                           for sb in sbs]))
        self.prm = {k: per(lambda sb, k=k: float(getattr(sb, k))) for k in self.NAMES}
        self.dt, self.L, self.g = (per(f) for f in (lambda sb: float(sb.time_dt), lambda sb: sb.L,
                                                    lambda sb: sb.g))
        self.r = _t(np.concatenate([sb.radius for sb in sbs]))[:, None]
        self.fixed = _t(np.concatenate([sb.fixvel for sb in sbs]))[:, None]
        self.m = 4.0 / 3.0 * math.pi * self.r ** 3 * self.prm["rho"]
        self.periodic = [self.sb.periodic in (1, 2), self.sb.periodic == 1, False]
        a, b, base = [], [], 0
        for sb in sbs:
            # pairs that can come into reach: at their speeds, gravity's and
            # what the overlaps at the start can add
            T, L = steps * sb.time_dt, [float(v) for v in sb.L]
            x, r = _t(sb.x - sb.origo), _t(sb.radius)[:, None]
            pa, pb = _pairs(x, r, x, r, L, [False] * 3, 0.0, True)
            over = r[pa] + r[pb] - torch.sqrt(_dot(x[pa] - x[pb], x[pa] - x[pb]))
            spring = math.sqrt(sb.k_n / (sb.rho * 4.0 * float(sb.radius.min()) ** 3))
            speed = (float(np.sqrt((sb.vel ** 2).sum(axis=1)).max()) + 10.0 * T
                     + spring * (float(over.max()) if len(over) else 0.0))
            pa, pb = _pairs(x, r, x, r, L, self.periodic,
                            2.0 * speed * T + 0.01 * float(sb.radius.max()) + sb.db, True)
            a.append(pa + base)
            b.append(pb + base)
            base += sb.np
        self.a, self.b = torch.cat(a), torch.cat(b)
        self.cost = len(self.r) + 3 * len(self.a)

    def start(self):
        cat = lambda k: _t(np.concatenate([getattr(sb, k) for sb in self.sbs]))  # noqa: E731
        n = len(self.r)
        st = {"x": cat("x"), "v": cat("vel"), "w": cat("angvel"), "angpos": cat("angpos"),
              "xysum": cat("xysum"), "h": torch.zeros((len(self.a), 3), dtype=torch.float64, device=_dev())}
        st["v0"], st["w0"] = st["v"], st["w"]
        st["es"] = st["ev"] = torch.zeros((n, 1), dtype=torch.float64, device=_dev())
        if self.sb.nw:
            st["wall"] = [float(self.sb.w_x[0]), float(self.sb.w_vel[0]), float(self.sb.w_vel[0]), 0.0]
        if self.sb.nb0:
            k = self.sb.nb0
            st["bond"] = torch.ones((k, 1), dtype=torch.bool, device=_dev())
            st["bd"] = st["bo"] = torch.zeros((k, 4), dtype=torch.float64, device=_dev())
        return st

    def length(self, v):
        d2 = _dot(v, v)
        # the floor keeps the derivative at zero finite
        return torch.sqrt(d2.clamp(min=1e-300)) if self.smooth else torch.sqrt(d2.float()).double()

    def root(self, v):
        return torch.sqrt(v) if self.smooth else torch.sqrt(v.float()).double()

    def slide(self, vt, lt, visc, still, moving, fn):
        """Viscous tangential force, limited by friction."""
        lim = torch.where(lt > 0.001, moving, still) * fn
        return torch.where(lt > 0.0, -torch.minimum(visc * lt, lim) * vt / lt.clamp(min=1e-300), 0.0 * vt)

    def contacts(self, st, prm, F, T, p, es, ev):
        h = st["h"]
        d = st["x"][self.a] - st["x"][self.b]
        for q in range(3):
            if self.periodic[q]:
                lq = self.L[self.a, q]
                d = torch.cat([d[:, k:k + 1] if k != q else
                               (d[:, q] - lq * torch.round(d[:, q] / lq))[:, None] for k in range(3)], 1)
        ln = self.length(d)
        gap = ln - (self.r[self.a] + self.r[self.b])
        model = self.sb.contactmodel
        hit = torch.nonzero((gap < (prm["db"][self.a] if model == 1 else 0.0))[:, 0])[:, 0]
        a, b = self.a[hit], self.b[hit]
        P = {k: v[a] for k, v in prm.items()}
        ra, rb, delta, n = self.r[a], self.r[b], gap[hit], d[hit] / ln[hit]
        dt = self.dt[a]
        vl = st["v"][a] - st["v"][b]
        vel = vl + (ra + delta / 2.0) * _cross(n, st["w"][a]) + (rb + delta / 2.0) * _cross(n, st["w"][b])
        vt = vel - n * _dot(n, vel)
        lt = self.length(vt)
        vn = _dot(vl, n) if model == 1 else -_dot(vl, n)
        fn = torch.clamp(-P["k_n"] * delta - P["gamma_n"] * vn, min=0.0) * n
        fc = -P["kappa"] * self.root(ra * rb) * n
        grip = self.length(fn - fc)
        if model == 1:
            ft = self.slide(vt, lt, P["gamma_t"], P["mu_s"], P["mu_d"], grip)
            ratio = torch.maximum(ra / rb, rb / ra)
            lam = -float(np.float32(0.9)) * self.root(ratio) * self.root(P["V_b"] / (2.0 * ra * rb / (ra + rb)))
            bridge = torch.exp((-delta / lam).float().double()).float().double()
            touch = delta < 0.0
            f = torch.where(touch, fn + ft + fc, -P["kappa"] * self.root(ra * rb) * bridge * n)
            press = torch.where(touch, self.length(fn), 0.0 * lt)
            return (F.index_add(0, a, f), T, p.index_add(0, a, press / (4.0 * math.pi * ra * ra)), es, ev, h)
        mu_s = 0.5 * (prm["mu_s"][a] + prm["mu_s"][b]) if self.smooth else P["mu_s"]
        mu_d = mu_s if self.smooth else P["mu_d"]
        h0 = h[hit]
        h0 = h0 - n * _dot(n, h0)
        hist = h0 + vt * dt
        ft = -P["k_t"] * hist - P["gamma_t"] * vt
        lf = self.length(ft)
        slip = lf > mu_s * grip
        t = ft / lf.clamp(min=1e-150)
        hist = torch.where(slip, -1.0 / P["k_t"] * (mu_d * grip * t + P["gamma_t"] * vt), hist)
        ft = torch.where(slip, mu_s * grip * t, ft)
        lever = -(ra + delta * 0.5) * n
        new = torch.zeros_like(h).index_add(0, hit, hist)
        F, T = F.index_add(0, a, fn + ft + fc), T.index_add(0, a, _cross(lever, ft))
        if not self.smooth:
            rate = torch.where(slip, self.length(self.length(ft) * vt * dt) / dt, 0.0 * lt)
            p = p.index_add(0, a, self.length(fn) / (4.0 * math.pi * ra * ra))
            es, ev = es.index_add(0, a, rate), ev.index_add(0, a, P["gamma_n"] * vn * vn)
        return F, T, p, es, ev, new

    def walls(self, st, prm, F, T, p):
        x, r, L = st["x"], self.r, self.L
        moving = st.get("wall")
        sides = [(2, -1.0, moving[0] if moving else L[:, 2:3], moving[1] if moving else 0.0), (2, 1.0, 0.0, 0.0)]
        if not self.periodic[0]:
            sides += [(0, -1.0, L[:, 0:1], 0.0), (0, 1.0, 0.0, 0.0)]
        if not self.periodic[1]:
            sides += [(1, -1.0, L[:, 1:2], 0.0), (1, 1.0, 0.0, 0.0)]
        load = 0.0
        for k, (q, sign, at, speed) in enumerate(sides):
            gap = (at - (x[:, q:q + 1] + r)) if sign < 0.0 else (x[:, q:q + 1] - r - at)
            i = torch.nonzero((gap < 0.0)[:, 0])[:, 0]
            if not len(i):
                continue
            P = {key: v[i] for key, v in prm.items()}
            n = torch.zeros((len(i), 3), dtype=torch.float64, device=x.device)
            n[:, q] = sign
            vel = st["v"][i] + r[i] * _cross(n, st["w"][i]) + speed
            vn = _dot(vel, n)
            vt = vel - n * vn
            fn = torch.clamp(-P["k_n"] * gap[i] - P["gamma_wn"] * vn, min=0.0) * n
            ln = self.length(fn)
            ft = self.slide(vt, self.length(vt), P["gamma_wt"], P["mu_ws"], P["mu_wd"], ln)
            F, T = F.index_add(0, i, fn + ft), T.index_add(0, i, -r[i] * _cross(n, ft))
            p = p.index_add(0, i, ln / (4.0 * math.pi * r[i] ** 2))
            if k == 0:
                load = float(_dot(fn.detach(), n).sum())
        return F, T, p, load

    def bonds(self, st, F, T):
        sb = self.sb
        pair = torch.as_tensor(sb.bonds.astype(np.int64), device=_dev())
        live = torch.nonzero(st["bond"][:, 0])[:, 0]
        i, j = pair[live, 0], pair[live, 1]
        dt, v, w = sb.time_dt, st["v"], st["w"]
        rb = sb.lambda_bar * torch.minimum(self.r[i], self.r[j])
        area, inert = math.pi * rb ** 2, 0.25 * math.pi * rb ** 4
        d = st["x"][i] - st["x"][j]
        ln = self.length(d)
        over = torch.clamp(ln - (self.r[i] + self.r[j]), max=0.0)
        n = d / ln
        t0, n0 = st["bd"][live, :3], st["bd"][live, 3:]
        dd = (v[i] - v[j] + (self.r[i] + over / 2.0) * _cross(n, w[i]) + (self.r[j] + over / 2.0) * _cross(n, w[j])) * dt
        ddn = -_dot(dd, n)
        ddt = dd - n * _dot(n, dd)
        dn, dtt = n0 + ddn, t0 - n * _dot(n, t0) + ddt
        fn = (sb.k_n * area * dn + sb.gamma_n * ddn / dt) * n
        ft = -sb.k_t * area * dtt - sb.gamma_t * ddt / dt
        mn, o0 = -n, st["bo"][live, :3]
        do = (w[j] - w[i]) * dt
        don = _dot(do, mn)
        on, ot = st["bo"][live, 3:] + don, o0 - mn * _dot(o0, mn) + do - don * mn
        tn, tt = -sb.k_t * 2.0 * inert * on * mn, -sb.k_n * inert * ot
        sigma = self.length(fn) / area + self.length(tt) * rb / inert
        tau = self.length(ft) / area + self.length(tn) * rb / (2.0 * inert)
        hold = ((sigma < sb.sigma_b) & (tau < sb.tau_b))[:, 0]
        bond, bd, bo = st["bond"].clone(), st["bd"].clone(), st["bo"].clone()
        bond[live, 0] = hold
        live, i, j = live[hold], i[hold], j[hold]
        bd[live], bo[live] = torch.cat([dtt, dn], 1)[hold], torch.cat([ot, on], 1)[hold]
        f, t = (fn + ft)[hold], (tn + tt)[hold]
        F, T = F.index_add(0, i, f).index_add(0, j, -f), T.index_add(0, i, -t).index_add(0, j, t)
        return F, T, bond, bd, bo

    def step(self, st, **override):
        prm = dict(self.prm, **override)
        z3, z1 = torch.zeros_like(st["x"]), torch.zeros_like(self.r)
        F, T, p, es, ev, h = self.contacts(st, prm, z3, z3, z1, z1, z1)
        F, T, p, load = self.walls(st, prm, F, T, p)
        new = dict(st, h=h)
        if self.sb.nb0:
            F, T, new["bond"], new["bd"], new["bo"] = self.bonds(st, F, T)
        dt, held = self.dt, self.fixed > 0.0
        acc, spin = F / self.m + self.g, T / (2.0 / 5.0 * self.m * self.r ** 2)
        if bool(held.any()):
            spin = torch.where(held, 0.0 * spin, spin)
            flat = torch.cat([0.0 * acc[:, :2], acc[:, 2:] - self.g[:, 2:]], 1)
            acc = torch.where(held, flat, acc)
        x = st["x"]
        for q in range(2):
            if self.periodic[q]:
                lq = self.L[:, q]
                x = x.clone()
                x[:, q] = torch.where(x[:, q] < 0.0, x[:, q] + lq, x[:, q])
                x[:, q] = torch.where(x[:, q] > lq, x[:, q] - lq, x[:, q])
        v0, w0 = st["v0"] + acc * dt, st["w0"] + spin * dt
        new.update(v0=v0, w0=w0, x=x + v0 * dt, v=v0 + 0.5 * acc * dt, w=w0 + 0.5 * spin * dt,
                   angpos=st["angpos"] + w0 * dt, F=F, T=T, p=p, es_dot=es, ev_dot=ev,
                   es=st["es"] + es * dt, ev=st["ev"] + ev * dt)
        new["xysum"] = st["xysum"] + new["v"][:, :2] * dt
        if self.sb.nw:
            at, _, half, _ = st["wall"]
            sb = self.sb
            push = (load - float(sb.w_devs[0]) * float(sb.L[0]) * float(sb.L[1])) / float(sb.w_m[0])
            half += push * sb.time_dt
            new["wall"] = [at + half * sb.time_dt, half + 0.5 * push * sb.time_dt, half, load]
        return new

    def fields(self, st):
        four = lambda a, w=None: torch.cat([a, 0.0 * self.r if w is None else w], 1)  # noqa: E731
        out = {"x": four(st["x"], self.r), "vel": four(st["v"], self.fixed), "xysum": st["xysum"],
               "force": four(st["F"]), "torque": four(st["T"]), "angpos": four(st["angpos"]),
               "angvel": four(st["w"])}
        out.update({k: st[k][:, 0] for k in ("es_dot", "es", "ev_dot", "ev", "p")})
        if self.sb.nw:
            at, speed, _, load = st["wall"]
            out["walls_nx"] = _t([[*self.sb.w_n[0], at]])
            out["walls_mvfd"] = _t([[self.sb.w_m[0], speed, load, self.sb.w_devs[0]]])
        if self.sb.nb0:
            out["bonds_delta"], out["bonds_omega"] = st["bd"], st["bo"]
        return out


def _exact_adjoint(bed, case, seed):
    st = bed.start()
    n = len(bed.r)
    leaf = {k: torch.tensor(float(getattr(bed.sb, k)), dtype=torch.float64, device=_dev(), requires_grad=True)
            for k in ("k_n", "k_t", "gamma_n")}
    mu = bed.prm["mu_s"].clone().requires_grad_()
    x0, v0 = (st[k].clone().requires_grad_() for k in ("x", "v"))
    keys = ("x", "v", "w", "v0", "w0", "angpos", "h")

    def few(count, k_n, k_t, gamma_n, mu, *vals):
        s = dict(st, **dict(zip(keys, vals)))
        prm = {k: v.expand(n, 1) for k, v in (("k_n", k_n), ("k_t", k_t), ("gamma_n", gamma_n))}
        for _ in range(count):
            s = bed.step(s, mu_s=mu, **prm)
        return tuple(s[k] for k in keys)

    vals = tuple({"x": x0, "v": v0, "v0": v0}.get(k, st[k]) for k in keys)
    left = case["steps"]
    while left:
        count = min(left, 5)
        vals = checkpoint(few, count, *leaf.values(), mu, *vals, use_reentrant=False)
        left -= count
    xb, vb = (_t(a) for a in _seeds(case, seed))
    loss = (vals[0] * xb).sum() + (vals[1] * vb).sum()
    g = torch.autograd.grad(loss, [*leaf.values(), mu, x0, v0])
    four = lambda a, w: torch.cat([a.detach(), w], 1)  # noqa: E731
    return {"x": four(vals[0], bed.r), "vel": four(vals[1], bed.fixed), "k_n": float(g[0]), "k_t": float(g[1]),
            "gamma_n": float(g[2]), "mu": g[3][:, 0], "x0": g[4], "v0": g[5]}


class _Flow:
    """The Darcy flow on the cell grid with its ring of ghost nodes."""

    def __init__(self, bed, ds):
        sb = bed.sb
        self.bed, self.sb = bed, sb
        self.num = [int(v) for v in sb.num]
        nx, ny, nz = self.num
        self.d = [float(v) / k for v, k in zip(sb.L, self.num)]
        node = lambda a: _t(a).reshape((nz + 2, ny + 2, nx + 2) + a.shape[1:])  # noqa: E731
        self.f = {k: node(v) for k, v in ds.arrays().items()}
        self.f["Ss"].fill_(1.0)
        z, y, x = torch.meshgrid(*(torch.arange(k, dtype=torch.float64, device=_dev()) for k in (nz, ny, nx)),
                                 indexing="ij")
        self.at = torch.stack([(c.reshape(-1) + 0.5) * d for c, d in zip((x, y, z), self.d)], 1)
        self.R = 0.5 * min(self.d)
        R = torch.full((len(self.at), 1), self.R, dtype=torch.float64, device=_dev())
        self.node, self.grain = _pairs(self.at, R, _t(sb.x), bed.r, [float(v) for v in sb.L], bed.periodic,
                                       0.1 * float(sb.radius.max()), False)
        mean = float(np.sum(sb.radius)) / sb.np * 2.0
        self.factor = mean * mean / 180.0 * 1.0e-6
        self.first = True

    def ghosts(self):
        for f in self.f.values():
            f[1:-1, 1:-1, -1], f[1:-1, 1:-1, 0] = f[1:-1, 1:-1, 1].clone(), f[1:-1, 1:-1, -2].clone()
            f[1:-1, -1, 1:-1], f[1:-1, 0, 1:-1] = f[1:-1, 1, 1:-1].clone(), f[1:-1, -2, 1:-1].clone()
            f[-1, 1:-1, 1:-1], f[0, 1:-1, 1:-1] = f[1, 1:-1, 1:-1].clone(), f[-2, 1:-1, 1:-1].clone()

    def step(self, x):
        f, bed, R, dt = self.f, self.bed, self.R, self.sb.time_dt
        nx, ny, nz = self.num
        d = self.at[self.node] - x[self.grain]
        for q in range(3):
            if bed.periodic[q]:
                lq = float(self.sb.L[q])
                d[:, q] -= lq * torch.round(d[:, q] / lq)
        dd, r = bed.length(d), bed.r[self.grain]
        lens = (math.pi * (R + r - dd) ** 2 * (dd * dd + 2.0 * dd * r - 3.0 * r * r + 2.0 * dd * R
                                               + 6.0 * r * R - 3.0 * R * R)) / (12.0 * dd)
        part = torch.where((R - r < dd) & (dd < R + r), lens, 0.0 * lens)
        part = part + torch.where(dd <= R - r, 4.0 / 3.0 * math.pi * r ** 3, 0.0 * lens)
        cell = 4.0 / 3.0 * math.pi * R ** 3
        void = cell - torch.zeros((nx * ny * nz, 1), dtype=torch.float64, device=x.device).index_add(0, self.node, part)
        phi = (void / cell).clamp(0.1, 0.9).reshape(nz, ny, nx)
        mid = (slice(1, -1),) * 3
        f["dphi"][mid] = 0.0 if self.first else phi - f["phi"][mid]
        self.first = False
        f["phi"][mid] = phi
        K = phi ** 3 / (1.0 - phi) ** 2 * self.factor * 1000.0 * -float(self.sb.g[2]) / NU
        f["K"][mid] = K
        f["T"][mid] = K[..., None] * _t(self.d)
        self.ghosts()
        H, near = f["H"], 0.0
        for q, axis in enumerate((2, 1, 0)):
            for to in (-1, 1):
                T0, T1 = f["T"][mid][..., q], torch.roll(f["T"][..., q], -to, axis)[mid]
                term = 2.0 * T0 * T1 / (T0 + T1) * (torch.roll(H, -to, axis)[mid] - H[mid]) / self.d[q] ** 2
                if q == 2:
                    term[-1 if to == 1 else 0] = 0.0
                near = near + term
        pore = -sum(self.d) / 3.0 * f["dphi"][mid] / dt
        new = f["H_new"]
        new[mid] = (H[mid] + dt / (f["Ss"][mid] * math.prod(self.d)) * (near + f["W"][mid] + pore)).clamp(min=0.0)
        f["H"], f["H_new"] = new, H
        for q, axis in enumerate((2, 1, 0)):
            slope = (torch.roll(new, -1, axis)[mid] - torch.roll(new, 1, axis)[mid]) / (2.0 * self.d[q])
            f["dH"][mid + (q,)] = slope
            f["V"][mid + (q,)] = -K / NU * slope / phi

    def fields(self):
        return {k: self.f[k].reshape((-1,) + self.f[k].shape[3:]) for k in FLOW_FIELDS}
