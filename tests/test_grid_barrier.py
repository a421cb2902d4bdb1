"""The count of the barrier over a whole grid (sphere_b200/csrc/barrier_count.h),
on the host: every block of a round waits for the same number of arrivals, the
last one of its own round, past 2^32 arrivals and whatever the grid; and, on the
GPU, the cell lists of kernels whose counters pass 2^32."""
import ctypes as C
import random
import subprocess
from pathlib import Path

import numpy as np
import pytest

from helpers import OUTPUT_FIELDS, STATE_FIELDS, mismatches, run_oracle
from sphere_b200 import scenes
from sphere_b200.sphk import Simulation
from sphere_b200.state import config_from_spherebin, state_from_spherebin

ROOT = Path(__file__).resolve().parent.parent
HERE = Path(__file__).resolve().parent


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = tmp_path_factory.mktemp("barrier") / "libbarrier_check.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-I",
                    str(ROOT / "sphere_b200" / "csrc"), str(HERE / "barrier_check.cpp"),
                    "-o", str(out)], check=True)
    lib = C.CDLL(str(out))
    lib.barrier_start_c.restype = C.c_uint64
    lib.barrier_round_end_c.argtypes = [C.c_uint64, C.c_uint64, C.c_uint32]
    lib.barrier_round_end_c.restype = C.c_uint64
    lib.barrier_open_c.argtypes = [C.c_uint64, C.c_uint64]
    return lib


# grids of the lists' kernels, powers of two among them; where the counter stands
# when the launch begins, as a number of whole grids past its start
@pytest.mark.parametrize("grid", [1, 7, 128, 296, 391, 592, 4096])
@pytest.mark.parametrize("where", ["start", "around_2_32", "far"])
def test_every_block_waits_for_its_own_round(lib, grid, where):
    start = lib.barrier_start_c()
    rounds = {"start": 0, "around_2_32": max(0, (2 ** 32 - start) // grid - 2),
              "far": 2 ** 44 // grid}[where]
    rng = random.Random(grid)
    count = start + rounds * grid
    for _ in range(3):                      # launches
        before = [0] * grid
        for _ in range(5):                  # barriers of a launch
            first = count
            for b in rng.sample(range(grid), grid):
                before[b] = lib.barrier_round_end_c(before[b], count, grid)
                count += 1
            assert set(before) == {first + grid} == {count}
            assert not lib.barrier_open_c(count - 1, before[0])
            assert lib.barrier_open_c(count, before[0])
    if where == "around_2_32" and grid > 1:
        assert first < 2 ** 32 + 15 * grid and count > 2 ** 32


@pytest.mark.gpu
@pytest.mark.parametrize("span", [None, 1], ids=["one_kernel", "split"])
def test_lists_past_2_32_arrivals(oracle_libs, span):
    """A list in every step, made by as many blocks as there are: k_small's
    counter passes 2^32 at about list 20, k_rebuild's at about list 50."""
    sb = scenes.collision(n=1500, seed=41, vmax=3.0, box=(0.3, 0.3, 0.3))
    sb.num = np.array([135, 135, 135], dtype=np.uint32)
    fields = STATE_FIELDS + OUTPUT_FIELDS + ("contacts", "delta_t")
    with Simulation(config_from_spherebin(sb), verlet_skin=0.0, topo_span=span) as sim:
        sim.upload(state_from_spherebin(sb))
        lists = sim.stats()["cell_rebuilds"]
        sim.step(150)
        sim.sync()
        got, lists = sim.download(), sim.stats()["cell_rebuilds"] - lists
        _, perm, _, _ = sim.cells()
    assert lists > 80
    rc, want, orun = run_oracle(oracle_libs["orc"], sb, 150)
    assert rc == 0
    assert mismatches(got, want, fields) == []
    assert np.array_equal(perm, orun.perm)


@pytest.mark.gpu
def test_barrier_and_list_by_themselves(tmp_path):
    """Rounds of the barrier on the device past 2^32 arrivals, a block that never
    comes (the others give up after a second and report it), and the cell list's
    kernel afterwards: it makes nothing until the status has been cleared.  A
    launch whose blocks do not fit on the device together returns its error."""
    from sphere_b200 import build
    exe = tmp_path / "cell_list_driver"
    subprocess.run([build.NVCC, *build.ARCH, "-O2", "--fmad=false", "-std=c++17", "-I",
                    str(ROOT / "sphere_b200" / "csrc"), str(HERE / "cell_list_driver.cu"), "-o", str(exe)],
                   check=True)
    res = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert res.returncode == 0, res.stdout + res.stderr
    assert res.stdout.count(": ok") == 13, res.stdout
