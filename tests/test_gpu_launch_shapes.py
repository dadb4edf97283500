"""Launch shapes: a tuned class changes its relaxations only, and a forced block size that
is too small for a large system's layout is raised for evaluations as for relaxations."""
import ctypes

import numpy as np
import pytest

from conftest import grid_from_golden
from firecore_b200 import systems as S
from firecore_b200.world import DEFAULT_FLAGS, FireParams, World
from oracle import oracle as O

pytestmark = pytest.mark.gpu
FTOL = 1e-5


@pytest.fixture(scope="module")
def world():
    return World(0)


def test_tuning_leaves_evaluations_alone(world, golden):
    """100 atoms x 160 without a cutoff: two lanes per atom on the image rows would add in
    another order."""
    b = S.make_systems([100] * 160, 61, topo_mode=1, sigma=0.05)
    try:
        world.set_params(flags=DEFAULT_FLAGS, Rcut=-1.0)
        world.grid_upload(golden["C"], grid_from_golden(golden))
        world.upload(b)
        F = world.eval()[0]
        assert world.lib.mmff_set_tuning(3, 0, 1, 256, 2) == 0
        assert np.array_equal(F, world.eval()[0])
    finally:
        world.lib.mmff_set_tuning(3, -1, 1, 0, 0)
        world.set_params(flags=DEFAULT_FLAGS, Rcut=10.0)


@pytest.mark.parametrize("threads", [64, 128, 256])
def test_forced_small_blocks_take_large_systems(world, golden, threads):
    grid = grid_from_golden(golden)
    b = S.make_systems([700], 23, topo_mode=1, sigma=0.0, cell=(200.0, 200.0, 40.0))
    b.neighCell[:] = 0
    try:
        world.set_params(flags=DEFAULT_FLAGS, npbc=(0, 0, 0), Rcut=-1.0)
        world.set_fire(FireParams())
        world.grid_upload(golden["C"], grid)
        world.upload(b)
        Fo, _ = O.eval_forces(b, O.make_params(grid, flags=DEFAULT_FLAGS, npbc=(0, 0, 0), Rcut=-1.0), golden["C"],
                              pos=world.state()["pos"])
        world.set_launch(threads, 0)
        F = world.eval()[0]
        assert np.abs(F - Fo).max() <= FTOL * np.abs(Fo).max()
        world.relax(1, 0.0, conv_mode=1)
        assert world.lib.mmff_get_forces(F.ctypes.data_as(ctypes.c_void_p)) == 0
        assert np.abs(F - Fo).max() <= FTOL * np.abs(Fo).max()
    finally:
        world.set_launch(0, 0)
        world.set_params(flags=DEFAULT_FLAGS, Rcut=10.0)


def test_autotune_of_few_large_systems(world, golden):
    """Half as many systems as SMs and fewer: candidates are timed in the form that runs (a
    cluster of blocks), every one of them launchable, and the relaxation goes on as before."""
    b = S.make_systems([100, 120, 300, 350], 67, topo_mode=1, sigma=0.1)
    try:
        world.set_params(flags=DEFAULT_FLAGS, Rcut=10.0)
        world.set_fire(FireParams())
        world.grid_upload(golden["C"], grid_from_golden(golden))
        world.upload(b)
        world.relax(40, 0.0, conv_mode=1)
        want = world.state()["pos"]
        world.restore()
        rep = world.autotune(nstep_probe=10)
        assert len(rep) and all(r["us_per_system_step"] > 0 for r in rep)
        world.relax(40, 0.0, conv_mode=1)
        assert np.array_equal(want, world.state()["pos"])
    finally:
        for c in range(6):
            world.lib.mmff_set_tuning(c, -1, 1, 0, 0)
