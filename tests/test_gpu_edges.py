"""Edges of the kernels' tiles and buffers: the radix sort's tile and digit
sizes, the porosity's per-plane hit buffer and grids of one to three cells an
axis, and differentiable sessions whose kept arrays are taken up again or
replaced."""
import ctypes as C

import numpy as np
import pytest

from helpers import BOND_FIELDS, OUTPUT_FIELDS, STATE_FIELDS, mismatches, run_oracle
from sphere_b200 import scenes, sphk
from sphere_b200.sphk import Simulation
from sphere_b200.spherebin import Spherebin
from sphere_b200.state import config_from_spherebin, state_from_spherebin
from test_darcy import NU, darcy_mismatches, run_darcy_oracle, seeded_grid

pytestmark = pytest.mark.gpu


# a tile is 1024 particles up to 148 x 1024, 4096 beyond; ids take one pass of
# up to 10 bits or two of up to 10
@pytest.mark.parametrize("num", [(1, 1, 1), (3, 11, 31), (4, 16, 16), (1, 1024, 1), (64, 64, 128)],
                         ids=lambda v: str(v[0] * v[1] * v[2]))
@pytest.mark.parametrize("n", [1, 31, 1024, 1025, 148 * 1024, 148 * 1024 + 1, 300001])
def test_noalloc_cell_list_at_tile_and_digit_edges(n, num):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(n + num[0])
    cell = 4e-3
    x = rng.uniform(-0.5 * cell, 1.0, (n, 4)) * np.array([num[0] * cell, num[1] * cell, num[2] * cell, 1e-3])
    sb = Spherebin(np_=1, nw=0)
    sb.L, sb.num, sb.time_dt = cell * np.array(num, float), np.array(num, dtype=np.uint32), 1.0
    conf = sphk.make_config(config_from_spherebin(sb))
    conf.np = n
    ncells = num[0] * num[1] * num[2]
    dev = torch.tensor(x, device="cuda")
    out = [torch.full((k,), 7, dtype=torch.int32, device="cuda") for k in (n, n, ncells, ncells)]
    lib = sphk.load_library()
    rc = lib.sph_cell_list_noalloc(C.byref(conf), C.c_void_p(dev.data_ptr()),
                                   *(C.c_void_p(o.data_ptr()) for o in out),
                                   C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0
    got = [o.cpu().numpy().view(np.uint32) for o in out]
    # calcCellID with the device's saturating conversion, ids past the grid last
    f = np.maximum(np.floor(x[:, :3] / (sb.L / np.array(num))), 0.0).astype(np.int64)
    c = (f[:, 2] * num[1]) * num[0] + f[:, 1] * num[0] + f[:, 0]
    c = np.where(c < ncells, c, ncells)
    perm = np.argsort(c, kind="stable")
    ids = c[perm]
    assert np.array_equal(got[1], perm.astype(np.uint32))
    assert np.array_equal(got[0], np.where(ids < ncells, ids, 0xFFFFFFFF).astype(np.uint32))
    lo = np.searchsorted(ids, np.arange(ncells), "left")
    hi = np.searchsorted(ids, np.arange(ncells), "right")
    assert np.array_equal(got[2], np.where(lo < hi, lo, 0xFFFFFFFF).astype(np.uint32))
    assert np.array_equal(got[3], np.where(lo < hi, hi, 0).astype(np.uint32))


@pytest.mark.parametrize("num", [(5, 5, 5), (2, 3, 4), (1, 2, 3), (33, 2, 1)],
                         ids=lambda v: "x".join(map(str, v)))
@pytest.mark.parametrize("periodic", [0, 1, 2])
def test_darcy_with_many_grains_a_cell(oracle_libs, num, periodic):
    """Coarse fluid grids: up to hundreds of grains overlap a cell's sphere,
    many times the porosity's buffer, and periodic neighbours repeat."""
    sb = scenes.collision(n=1100, seed=17, periodic=periodic, k_n=500.0, k_t=500.0, vmax=0.1)
    sb.num = np.array(num, dtype=np.uint32)
    start = seeded_grid(sb.num, 5)
    _, so, o = run_darcy_oracle(oracle_libs["orc"], sb, 6, start.copy())
    with Simulation(config_from_spherebin(sb)) as sim:
        sim.upload(state_from_spherebin(sb))
        sim.darcy_upload(start.copy(), NU)
        sim.step(2)
        sim.step(4)
        sim.sync()
        st, g = sim.download(), sim.darcy_download()
    assert darcy_mismatches(g, o) == []
    assert mismatches(st, so, STATE_FIELDS) == []


# a block of 128 grains an SM (148 of them): beside a flow the step in one kernel,
# and past it split
@pytest.mark.parametrize("n", [18944, 18945])
def test_darcy_at_the_largest_scene_in_one_kernel(oracle_libs, n):
    sb = scenes.collision(n=n, seed=29, box=(0.1, 0.1, 0.1), k_n=500.0, k_t=500.0, vmax=0.5)
    sb.num = np.array([16, 16, 16], dtype=np.uint32)
    start = seeded_grid(sb.num, 7)
    _, so, o = run_darcy_oracle(oracle_libs["orc"], sb, 4, start.copy())
    with Simulation(config_from_spherebin(sb)) as sim:
        sim.upload(state_from_spherebin(sb))
        sim.darcy_upload(start.copy(), NU)
        sim.step(4)
        sim.sync()
        st, g = sim.download(), sim.darcy_download()
    assert darcy_mismatches(g, o) == []
    assert mismatches(st, so, STATE_FIELDS) == []


def test_sessions_take_up_kept_arrays_or_replace_them():
    """Differentiable sessions of one context: the same checkpoint interval
    again, another, the first again, with plain steps and another scene's
    state between them, give what a context of their own gives."""
    scene = {k: scenes.collision(n=300, seed=k, vmax=0.2, wmax=50.0) for k in (3, 4)}
    w = np.random.default_rng(8).normal(size=(300, 3))

    def session(sim, sb, every):
        sim.upload(state_from_spherebin(sb))
        sim.diff_begin(checkpoint_every=every)
        sim.step(17)
        sim.sync()
        x = sim.download().x
        g = sim.diff_backward(w, 1e-3 * w)
        sim.diff_end()
        return x, g

    with Simulation(config_from_spherebin(scene[3])) as sim:
        for seed, every in ((3, 5), (4, 5), (3, 8), (3, 5)):
            x, g = session(sim, scene[seed], every)
            sim.step(3)
            sim.sync()
            with Simulation(config_from_spherebin(scene[seed])) as own:
                x_own, g_own = session(own, scene[seed], every)
            assert np.array_equal(x, x_own)
            # only the order of atomic additions may differ
            for k in ("k_n", "k_t", "gamma_n"):
                assert abs(g[k] - g_own[k]) <= 1e-11 * abs(g_own[k]), (k, seed, every)
            assert np.allclose(g["x0"], g_own["x0"], rtol=1e-9, atol=1e-12 * np.abs(g_own["x0"]).max())


def test_a_kept_tape_gives_way_to_a_session_that_needs_the_memory():
    """With less of the device free than a tape takes, a context's session gets the
    tape that another context has kept since its own ended; that one's next session
    allocates anew."""
    torch = pytest.importorskip("torch")
    sb = scenes.collision(n=4000, seed=3, vmax=0.2, wmax=50.0)
    w = np.random.default_rng(8).normal(size=(4000, 3))

    def session(sim):
        sim.upload(state_from_spherebin(sb))
        sim.diff_begin(checkpoint_every=64)
        sim.step(20)
        sim.sync()
        g = sim.diff_backward(w, 1e-3 * w)
        sim.diff_end()
        return g

    with Simulation(config_from_spherebin(sb)) as a, Simulation(config_from_spherebin(sb)) as b:
        b.upload(state_from_spherebin(sb))
        alone = a.stats()["device_bytes"]
        first = session(a)
        kept = a.stats()["device_bytes"] - alone
        assert kept > 250e6   # 64 rows of 4000 particles, 1 KB each
        torch.cuda.synchronize()
        free, _ = torch.cuda.mem_get_info()
        fill = torch.empty(free - int(0.8 * kept), dtype=torch.uint8, device="cuda")
        second = session(b)
        assert a.stats()["device_bytes"] - alone < 0.2 * kept
        del fill
        torch.cuda.empty_cache()
        third = session(a)
    for g in (second, third):
        for k in ("k_n", "k_t", "gamma_n"):   # only the order of atomic additions may differ
            assert abs(g[k] - first[k]) <= 1e-11 * abs(first[k])


# the terms the linear law leaves out: the capillary force where kappa is 0
# (either sign), lengths only compared with zero (velocities 0, below and
# above the smallest float square), the pressure of steps inside a call
@pytest.mark.parametrize("kappa", [0.0, -0.0, 1e-3])
@pytest.mark.parametrize("speed", [0.0, 1e-24, 1e-21, 0.3])
@pytest.mark.parametrize("span", [None, 1], ids=["one_kernel", "split"])
def test_linear_law_leaves_out_only_what_changes_nothing(oracle_libs, kappa, speed, span):
    sb = scenes.collision(n=400, seed=23, vmax=speed, wmax=100.0 * speed, mu=0.0 if speed == 1e-21 else 0.4,
                          g=(0.0, 0.0, 0.0))
    sb.kappa = kappa
    cfg = config_from_spherebin(sb)
    fields = STATE_FIELDS + OUTPUT_FIELDS + ("contacts", "delta_t")
    with Simulation(cfg, topo_span=span) as sim:
        sim.upload(state_from_spherebin(sb))
        done = 0
        for k in (1, 3, 8, 11):
            sim.step(k)
            sim.sync()
            done += k
            rc, want, _ = run_oracle(oracle_libs["orc"], sb, done)
            assert rc == 0
            assert mismatches(sim.download(), want, fields) == [], done


# grains on the vertices of the grid, a few units in the last place and 2^-20
# of a cell to either side: the cell of a position beside a boundary
@pytest.mark.parametrize("span", [None, 1], ids=["one_kernel", "split"])
@pytest.mark.parametrize("num, L, origo", [((7, 11, 13), (0.1, 0.2, 0.3), (0.0, 0.0, 0.0)),
                                           ((9, 5, 6), (0.07, 0.011, 1.3), (0.013, 0.001, 0.1)),
                                           ((4, 4, 8), (1.0, 1.0, 2.0), (0.0, 0.0, 0.0))])
def test_cells_of_positions_at_cell_boundaries(oracle_libs, num, L, origo, span):
    rng = np.random.default_rng(num[0])
    k = np.stack(np.meshgrid(*(np.arange(1, m) for m in num), indexing="ij"), -1).reshape(-1, 3)
    cell = np.array(L) / np.array(num)
    x = np.array(origo) + k * cell
    side = rng.integers(-3, 4, x.shape)
    x = x + side * np.spacing(np.abs(x))
    far = rng.random(x.shape) < 0.3
    x = np.where(far, x + side * 2.0 ** -21 * cell, x)
    x = x[np.all(x < np.array(L) - 1e-4, axis=1)]   # clear of the default walls at L
    sb = scenes.collision(n=len(x), seed=1, vmax=0.0, wmax=0.0, g=(0.0, 0.0, 0.0))
    sb.x, sb.radius = x, np.full(len(x), 1e-5)
    sb.origo, sb.L, sb.num = np.array(origo), np.array(L), np.array(num, dtype=np.uint32)
    rc, want, orun = run_oracle(oracle_libs["orc"], sb, 5)
    with Simulation(config_from_spherebin(sb), topo_span=span) as sim:
        sim.upload(state_from_spherebin(sb))
        sim.step(5)
        sim.sync()
        got = sim.download()
        cell_sorted, perm, _, _ = sim.cells()
    assert rc == 0 and mismatches(got, want, STATE_FIELDS + OUTPUT_FIELDS) == []
    assert np.array_equal(perm, orun.perm) and np.array_equal(cell_sorted, orun.cell_sorted)


# the bonds' screens: viscous terms that are there or not, strengths that some
# bonds, all and none reach, and strengths outside the screen's range
@pytest.mark.parametrize("gamma_n, gamma_t", [(0.0, 0.0), (3.0, 0.0), (0.0, 2.0), (3.0, 2.0), (-0.0, -0.0)])
@pytest.mark.parametrize("sigma_b, tau_b", [(3e-3, 3e-3), (1.0, 1e-3), (1e-130, 1e-130), (1e130, 1e130),
                                            (np.inf, np.inf), (-1.0, 1.0)])
def test_bond_breaking_and_viscosity(oracle_libs, gamma_n, gamma_t, sigma_b, tau_b):
    sb = scenes.tension(nx=7, ny=4, nz=5, seed=3, sigma_b=sigma_b, tau_b=tau_b)
    sb.gamma_n, sb.gamma_t = gamma_n, gamma_t
    rc, want, _ = run_oracle(oracle_libs["orc"], sb, 120)
    assert rc == 0
    with Simulation(config_from_spherebin(sb)) as sim:
        sim.upload(state_from_spherebin(sb))
        sim.step(120)
        sim.sync()
        assert mismatches(sim.download(), want, STATE_FIELDS + OUTPUT_FIELDS + BOND_FIELDS) == []
