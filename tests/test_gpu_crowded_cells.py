"""Cells with many members: the cell list's order from two members a cell to all
grains in one (past 16,384 a block looks for them in index order), the bucket of
the outside among them, and steps over such cells against the oracle."""
import numpy as np
import pytest

from helpers import OUTPUT_FIELDS, STATE_FIELDS, mismatches, run_oracle
from sphere_b200 import scenes
from sphere_b200.spherebin import Spherebin
from sphere_b200.sphk import BatchSimulation, SphError, Simulation
from sphere_b200.state import config_from_spherebin, state_from_spherebin

pytestmark = pytest.mark.gpu

ALL = STATE_FIELDS + OUTPUT_FIELDS + ("contacts", "delta_t")


def _cloud(n, num):
    sb = Spherebin(np_=n, nw=0)
    sb.L, sb.num = np.array([0.1, 0.1, 0.1]), np.array(num, dtype=np.uint32)
    sb.x, sb.radius = np.random.default_rng(2).uniform(0.0, 0.1, (n, 3)), np.full(n, 1e-6)
    sb.time_dt = 1e-6
    return sb


@pytest.mark.parametrize("outside", [0.0, 0.5, 1.0])
@pytest.mark.parametrize("n, num", [(33, (1, 1, 1)), (5000, (2, 1, 1)), (16384, (1, 1, 1)),
                                    (16385, (1, 1, 1)), (70000, (1, 1, 1)), (200000, (3, 1, 1)), (300000, (18, 1, 1)), (300000, (40, 40, 40))],
                         ids=lambda v: str(v if isinstance(v, int) else v[0] * v[1] * v[2]))
def test_order_of_crowded_cells(n, num, outside):
    sb = _cloud(n, num)
    out = np.random.default_rng(3).random(n) < outside
    sb.x[out, 2] = 1.0   # above the grid: past the last cell
    f = np.floor(sb.x / (sb.L / np.array(num))).astype(np.int64)
    ncells = int(np.prod(num))
    cell = np.minimum((f[:, 2] * num[1] + f[:, 1]) * num[0] + f[:, 0], ncells)
    perm = np.argsort(cell, kind="stable")
    with Simulation(config_from_spherebin(sb)) as sim:
        if out.any():
            with pytest.raises(SphError, match="OUT_OF_GRID"):
                sim.upload(state_from_spherebin(sb))
        else:
            sim.upload(state_from_spherebin(sb))
        ids, got, _, _ = sim.cells()
    assert np.array_equal(got, perm.astype(np.uint32))
    assert np.array_equal(ids, np.where(cell[perm] < ncells, cell[perm], 0xFFFFFFFF).astype(np.uint32))


@pytest.mark.parametrize("span", [None, 1], ids=["one_kernel", "split"])
@pytest.mark.parametrize("skin", [0.0, 0.1])
def test_steps_with_ten_thousand_grains_in_a_cell(oracle_libs, span, skin):
    sb = scenes.collision(n=10000, seed=19, r=(0.3e-3, 0.5e-3), vmax=2.0, k_n=500.0, k_t=500.0)
    sb.num = np.array([1, 1, 1], dtype=np.uint32)
    rc, want, orun = run_oracle(oracle_libs["orc"], sb, 4)
    assert rc == 0
    with Simulation(config_from_spherebin(sb), verlet_skin=skin, topo_span=span) as sim:
        sim.upload(state_from_spherebin(sb))
        sim.step(4)
        sim.sync()
        got = sim.download()
        _, perm, _, _ = sim.cells()
    assert mismatches(got, want, ALL) == []
    assert np.array_equal(perm, orun.perm)


@pytest.mark.parametrize("span", [None, 1], ids=["one_kernel", "split"])
def test_a_scene_of_a_batch_that_left_its_grid(oracle_libs, span):
    """Its 6,000 grains share the bucket of the outside in every step; the other
    scenes go on."""
    sbs = [scenes.collision(n=n, seed=n, vmax=1.0) for n in (700, 6000, 900)]
    sbs[1].vel[:, 2] = 2e5   # out of the grid in the first step
    with BatchSimulation([config_from_spherebin(sb) for sb in sbs], topo_span=span) as sim:
        sim.upload([state_from_spherebin(sb) for sb in sbs])
        sim.step(40)
        with pytest.raises(SphError, match="OUT_OF_GRID"):
            sim.sync()
        got = sim.download_all()
    for sb, st in zip(sbs[::2], got[::2]):
        rc, want, _ = run_oracle(oracle_libs["orc"], sb, 40)
        assert rc == 0
        assert mismatches(st, want, ALL) == []
