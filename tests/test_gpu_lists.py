"""The candidate lists across changes of cell: grains that cross cells while
their lists stay in use, several new contacts of one grain in one step (whose
slots follow the reference's visiting order), cells of every size against the
reach of a list, grids of two and three periodic cells, lists that overflow
and grains outside their cells' boxes.  Everything bit for bit against the
oracle, the cell list of the last step included.  Each with the step in one
kernel, as scenes of this size run, and in the split kernels of larger ones
(which asking for a search span selects)."""
import numpy as np
import pytest

from helpers import OUTPUT_FIELDS, STATE_FIELDS, WALL_FIELDS, mismatches, run_oracle, with_model
from sphere_b200 import scenes
from sphere_b200.sphk import BatchSimulation, Simulation
from sphere_b200.state import config_from_spherebin, state_from_spherebin

pytestmark = pytest.mark.gpu

ALL = STATE_FIELDS + OUTPUT_FIELDS + ("contacts", "delta_t") + WALL_FIELDS


def _flow(cell, periodic, n=900, seed=91, r=(0.8e-3, 1.6e-3), nw=0, **kw):
    """Soft grains in fast motion; cells `cell` times the largest radius wide."""
    sb = scenes.collision(n=n, seed=seed, periodic=periodic, r=r, nw=nw, vmax=6.0, k_n=500.0,
                          k_t=500.0, gamma_n=0.01, straddle=periodic != 0, **kw)
    sb.num = np.maximum(1, np.floor(sb.L / (cell * r[1]))).astype(np.uint32)
    return sb


SCENES = {
    # two radii a cell: pairs of a list can be two cells apart
    "cells_2r": lambda: _flow(2.0, 0),
    "cells_2r_periodic": lambda: _flow(2.0, 1, box=(0.032, 0.032, 0.06)),
    "cells_2r_periodic_x": lambda: _flow(2.0, 2, box=(0.032, 0.06, 0.06)),
    # cells that hold the whole reach of a list
    "cells_3r": lambda: _flow(3.0, 0, nw=1),
    # below a diameter: overlapping grains the stencil does not reach
    "cells_1.5r": lambda: _flow(1.5, 0),
    # too small for any list to outlive a change of cell
    "cells_1.05r": lambda: _flow(1.05, 0, n=500),
    # three and two cells around a periodic axis
    "three_cells": lambda: _flow(3.0, 1, n=400, box=(0.0165, 0.0165, 0.05)),
    "two_cells": lambda: _flow(4.5, 1, n=400, box=(0.0165, 0.0165, 0.05)),
    # grains four times their neighbours' size: more candidates than a list holds
    "overflow": lambda: _flow(2.0, 0, n=1200, r=(0.35e-3, 2.0e-3)),
    # and among them grains that cross a side
    "overflow_periodic": lambda: _few_large(),
}


def _few_large():
    """A sheared periodic bed of fine grains with a few large ones, whose candidates
    are more than a list holds in nearly every step."""
    sb = _sheared(n=1500, seed=12)
    r = 0.4 * sb.radius
    r[np.random.default_rng(12).choice(1500, 12, replace=False)] = 2.6e-3
    sb.radius = r
    sb.num = np.maximum(3, np.floor(sb.L / 5.2e-3)).astype(np.uint32)
    return sb


both_kernels = pytest.mark.parametrize("span", [None, 1], ids=["one_kernel", "split"])


@both_kernels
@pytest.mark.parametrize("name", sorted(SCENES))
@pytest.mark.parametrize("skin", [0.1, 0.5])
def test_lists_outlive_changes_of_cell(oracle_libs, name, skin, span):
    sb = SCENES[name]()
    rc, want, orun = run_oracle(oracle_libs["orc"], sb, 90)
    assert rc == 0
    cfg = config_from_spherebin(sb)
    with Simulation(cfg, verlet_skin=skin, topo_span=span) as sim:
        sim.upload(state_from_spherebin(sb))
        for k in (33, 1, 56):
            sim.step(k)
        sim.sync()
        got = sim.download()
        cell_sorted, perm, cstart, cend = sim.cells()
    assert mismatches(got, want, ALL) == []
    assert np.array_equal(perm, orun.perm) and np.array_equal(cell_sorted, orun.cell_sorted)
    assert np.array_equal(cstart, orun.cell_start)
    occ = orun.cell_start != 0xFFFFFFFF
    assert np.array_equal(cend[occ], orun.cell_end[occ])


@both_kernels
@pytest.mark.parametrize("db, V_b, kappa", [(1e-4, 1e-12, 0.05), (1.2e-3, 1e-9, 1e-3)], ids=["near", "far"])
@pytest.mark.parametrize("name", ["cells_2r", "cells_2r_periodic", "cells_1.5r", "two_cells"])
def test_model1_lists_outlive_changes_of_cell(oracle_libs, name, db, V_b, kappa, span):
    """Contact model 1 sums its pairs in visiting order: the order of a list
    follows the grains' present cells.  With the wide reach some grains have
    more acting pairs than a list, or the warp's shared memory, holds."""
    sb = with_model(SCENES[name](), 1, kappa=kappa, V_b=V_b, db=db)
    rc, want, _ = run_oracle(oracle_libs["orc"], sb, 60)
    assert rc == 0
    with Simulation(config_from_spherebin(sb), verlet_skin=0.3, topo_span=span) as sim:
        sim.upload(state_from_spherebin(sb))
        sim.step(60)
        sim.sync()
        got = sim.download()
    assert mismatches(got, want, ALL) == []


@both_kernels
def test_batched_scenes_of_either_kind(oracle_libs, span):
    """Scenes whose lists outlive changes of cell beside scenes whose do not."""
    sbs = [SCENES[k]() for k in ("cells_2r", "cells_1.05r", "two_cells", "cells_2r_periodic_x")]
    with BatchSimulation([config_from_spherebin(sb) for sb in sbs], verlet_skin=0.3,
                         topo_span=span) as sim:
        sim.upload([state_from_spherebin(sb) for sb in sbs])
        sim.step(50)
        sim.sync()
        got = sim.download_all()
    for sb, st in zip(sbs, got):
        rc, want, _ = run_oracle(oracle_libs["orc"], sb, 50)
        assert rc == 0
        assert mismatches(st, want, STATE_FIELDS + OUTPUT_FIELDS + ("contacts", "delta_t")) == []


@both_kernels
@pytest.mark.parametrize("fast", [0, 13, 31, 40])
def test_the_fastest_grain_of_a_split_warp_sets_the_clock(oracle_libs, fast, span):
    """One grain in motion among grains at rest, some of which touch walls or one
    another, so that its warp takes different ways to the displacement's maximum:
    it meets grains that were beyond its list's reach."""
    sb = scenes.collision(n=96, seed=7, vmax=0.0, wmax=0.0, g=(0.0, 0.0, 0.0), phi_target=0.2)
    lo = np.min(sb.x - sb.radius[:, None], axis=0)
    sb.x = sb.x - lo - 1e-5
    sb.L = np.max(sb.x + sb.radius[:, None], axis=0) - 1e-5
    sb.num = np.maximum(1, np.floor(sb.L / 3.3e-3)).astype(np.uint32)
    sb.vel[fast] = np.array([9.0, 7.0, 11.0]) * np.where(sb.x[fast] > 0.5 * sb.L, -1.0, 1.0)
    rc, want, _ = run_oracle(oracle_libs["orc"], sb, 120)
    assert rc == 0 and int((want.contacts != sb.np).sum()) > 0
    with Simulation(config_from_spherebin(sb), verlet_skin=0.05, topo_span=span) as sim:
        sim.upload(state_from_spherebin(sb))
        sim.step(120)
        sim.sync()
        assert mismatches(sim.download(), want, ALL) == []


def _crossing_pairs(periodic, reach, sides, seed):
    """Pairs in contact that travel out through a periodic side together or one
    after the other, at every phase against the cells of the other axis: some cross
    into the next cell in the step of their return."""
    rng = np.random.default_rng(seed)
    r, dt, num = 1e-3, 2e-6, 8 if reach == "one_image" else 3
    cell = 2.05e-3 if reach == "one_image" else 1.7e-3   # an axis of 5.1 mm: under 2.5 reaches
    L = num * cell
    x, vel = [], []
    for i in range(36):
        hi = sides == "upper" or (sides == "both" and i % 2 == 0)
        ax = (i // 2) % 2 if periodic == 1 else 0
        k = 3 + i                                  # the step that takes it out
        v = np.zeros(3)
        p = np.array([0.0, 0.0, 2.5e-3 + 4.6e-3 * i])
        v[ax] = 0.6 if hi else -0.6
        p[ax] = (L if hi else 0.0) - (k - 0.5) * dt * v[ax]
        v[1 - ax] = rng.choice([-0.7, 0.7])        # into the next cell one step later, or about then
        p[1 - ax] = cell * rng.integers(1, num) - (k + 0.5 + rng.choice([0.0, 0.0, 1.0, -1.0])) * dt * v[1 - ax]
        d = np.zeros(3)
        d[rng.integers(0, 3)] = 2 * r - 1e-7
        if d[ax] != 0.0 and hi:
            d = -d
        x += [p, p + d]
        vel += [v, v]
    sb = scenes.collision(n=len(x), seed=1, periodic=periodic, wmax=20.0, g=(0.0, 0.0, 0.0), dt=dt, k_n=500.0,
                          k_t=500.0, gamma_n=0.0)
    sb.L = np.array([L, L if periodic == 1 else 3 * L, 4.6e-3 * 37])
    sb.num = np.array([num, num if periodic == 1 else 3 * num, 78], dtype=np.uint32)
    sb.x, sb.vel, sb.radius = np.array(x) % np.where(np.arange(3) < 2, sb.L, 1e9), np.array(vel), np.full(len(x), r)
    return sb


@both_kernels
@pytest.mark.parametrize("reach", ["one_image", "short_axis"])
@pytest.mark.parametrize("periodic, sides", [(1, "upper"), (1, "lower"), (1, "both"), (2, "both")])
@pytest.mark.parametrize("seed", [1, 2])
def test_grains_that_cross_a_periodic_side(oracle_libs, periodic, sides, reach, seed, span):
    """The images of list entries and slots, and the lists recorded while a grain
    stood outside, with epochs that end in the steps of the crossings."""
    sb = _crossing_pairs(periodic, reach, sides, seed)
    rc, want, _ = run_oracle(oracle_libs["orc"], sb, 70)
    assert rc == 0 and int((want.contacts != sb.np).sum()) >= sb.np // 2
    for skin in (0.1, 0.01, 0.004):
        with Simulation(config_from_spherebin(sb), verlet_skin=skin, topo_span=span) as sim:
            sim.upload(state_from_spherebin(sb))
            for k in (20, 1, 49):
                sim.step(k)
            sim.sync()
            assert mismatches(sim.download(), want, ALL) == [], skin


def _sheared(n=1500, cell=2.0, seed=6, periodic=1):
    """A dense bed in fast shear: grains cross the sides in nearly every step, in a
    moving contact network."""
    side = (n * 8.2e-9 / 0.35) ** (1 / 3)
    sb = scenes.collision(n=n, seed=seed, periodic=periodic, box=(1.02 * side, 1.02 * side, 1.2 * side + 0.012),
                          phi_target=0.35, k_n=500.0, k_t=500.0, gamma_n=0.01, vmax=2.0, straddle=True)
    sb.vel = sb.vel + np.stack([6.0 * (2 * sb.x[:, 2] / sb.L[2] - 1), 0 * sb.x[:, 0], 0 * sb.x[:, 0]], 1)
    sb.num = np.maximum(1, np.floor(sb.L / (cell * 1.6e-3))).astype(np.uint32)
    return sb


@both_kernels
@pytest.mark.parametrize("model", [1, 2])
@pytest.mark.parametrize("cell", [2.0, 2.4, 3.0])
def test_sheared_beds_with_periodic_sides(oracle_libs, cell, model, span):
    sb = _sheared(cell=cell)
    if model == 1:
        sb = with_model(sb, 1, kappa=0.05, V_b=1e-12, db=1e-4)
    rc, want, orun = run_oracle(oracle_libs["orc"], sb, 150)
    assert rc == 0
    for kw in (dict(verlet_skin=0.1), dict(verlet_skin=0.3), dict(relayout_every=7, graph_steps=3)):
        with Simulation(config_from_spherebin(sb), topo_span=span, **kw) as sim:
            sim.upload(state_from_spherebin(sb))
            sim.step(150)
            sim.sync()
            got = sim.download()
            _, perm, _, _ = sim.cells()
        assert mismatches(got, want, ALL) == [], kw
        assert np.array_equal(perm, orun.perm)


@both_kernels
def test_batched_scenes_with_periodic_sides(oracle_libs, span):
    """Crossings of several scenes in a step, of scenes whose axes are too short to
    follow an image beside ones that do."""
    sbs = [_crossing_pairs(1, "one_image", "both", 3), _sheared(n=800, seed=7), _crossing_pairs(1, "short_axis", "both", 4),
           _sheared(n=700, seed=10, cell=2.4), _crossing_pairs(2, "one_image", "both", 5)]
    with BatchSimulation([config_from_spherebin(sb) for sb in sbs], topo_span=span) as sim:
        for _ in range(2):   # another run of the same context
            sim.upload([state_from_spherebin(sb) for sb in sbs])
            sim.step(70)
            sim.sync()
        got = sim.download_all()
    for sb, st in zip(sbs, got):
        rc, want, _ = run_oracle(oracle_libs["orc"], sb, 70)
        assert rc == 0
        assert mismatches(st, want, STATE_FIELDS + OUTPUT_FIELDS + ("contacts", "delta_t")) == []


def test_differentiable_steps_with_periodic_sides():
    """The forward with lists and with a sweep in every step, bit for bit."""
    sb = _sheared(n=900, seed=9)
    x = []
    for skin in (0.0, 0.1):
        with Simulation(config_from_spherebin(sb), verlet_skin=skin) as sim:
            sim.upload(state_from_spherebin(sb))
            sim.diff_begin(checkpoint_every=16)
            sim.step(120)
            sim.sync()
            x.append(sim.download())
            sim.diff_end()
    assert mismatches(x[1], x[0], STATE_FIELDS + ("force", "torque", "contacts", "delta_t")) == []


@both_kernels
@pytest.mark.parametrize("skin", [0.0, 0.1, 0.4])
@pytest.mark.parametrize("shift", [0.0, -0.07, 0.05])
@pytest.mark.parametrize("periodic", [0, 1])
def test_beds_that_stand_out_of_their_grid(oracle_libs, periodic, shift, skin, span):
    """Grains beyond the sides for the whole run, in cells that their ids saturate
    to or alias, some on their way in or out."""
    sb = scenes.settling(4, 11, 11, 6)
    sb.L, sb.num = np.array([0.2, 0.18, 2.0]), np.array([9, 8, 96], dtype=np.uint32)
    sb.periodic = periodic
    sb.x = sb.x + np.array([shift, 0.7 * shift, 0.02])
    sb.vel = np.random.default_rng(3).uniform(-3.0, 3.0, sb.x.shape) * np.array([1.0, 1.0, 0.2])
    rc, want, orun = run_oracle(oracle_libs["orc"], sb, 60)
    assert rc == 0
    with Simulation(config_from_spherebin(sb), verlet_skin=skin, topo_span=span) as sim:
        sim.upload(state_from_spherebin(sb))
        for k in (7, 53):
            sim.step(k)
        sim.sync()
        got = sim.download()
        _, perm, _, _ = sim.cells()
    assert mismatches(got, want, ALL) == []
    assert np.array_equal(perm, orun.perm)
