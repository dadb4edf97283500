"""Forces of the relaxation kernels themselves (one step from given positions)
against the FP64 oracle, at the sizes where their work split changes: i-blocks
of 32 atoms, chunks of 8 atoms j, a last block shared by 2, 4, ... lanes per
atom, every block size, with and without a cutoff (pair lists / all images in
the ordered loop), with and without H-bond pseudo-charges; pair lists against
per-step candidate rows; a system beyond the largest shared-memory layout.
Tolerance as for the evaluation: 1e-5 of the system's largest force."""
import ctypes

import numpy as np
import pytest

from conftest import grid_from_golden
from firecore_b200 import systems as S
from firecore_b200.world import DEFAULT_FLAGS, FireParams, World
from oracle import oracle as O

pytestmark = pytest.mark.gpu
SMALL = [20, 23, 24, 25, 31, 32, 33, 34, 35, 36, 37, 40, 41, 48, 49, 63, 64]
LARGE = [65, 66, 68, 72, 73, 96, 97, 104, 127, 128, 129, 131, 160, 200, 255, 256, 257, 300]
FTOL = 1e-5


@pytest.fixture(scope="module")
def world():
    return World(0)


def step_forces(w, b):
    """Forces of the first step of a relaxation."""
    w.restore()
    w.relax(1, 0.0, conv_mode=1)
    F = np.zeros((int(b.nvecs.sum()), 3))
    assert w.lib.mmff_get_forces(F.ctypes.data_as(ctypes.c_void_p)) == 0
    return F


def compare(b, F, Fo):
    a, n, v = b.offsets()
    checked = 0
    for s in range(b.nsys):
        ref = Fo[v[s]:v[s + 1]]
        if np.abs(ref).max() > 1e5:          # atoms on top of an image: the sums clamp such forces
            continue
        err = np.abs(F[v[s]:v[s + 1]] - ref).max() / np.abs(ref).max()
        assert err < FTOL, (int(b.natoms[s]), err)
        checked += 1
    assert checked >= 0.7 * b.nsys, checked


def batch(world, golden, sizes, rcut, hbond):
    grid = grid_from_golden(golden)
    b = S.make_systems(sizes, 17, topo_mode=1, sigma=0.05, hbond=hbond)
    world.set_params(flags=DEFAULT_FLAGS, Rcut=rcut)
    world.set_fire(FireParams())
    world.grid_upload(golden["C"], grid)
    world.upload(b)
    pos = world.state()["pos"]
    Fo, _ = O.eval_forces(b, O.make_params(grid, flags=DEFAULT_FLAGS, Rcut=rcut), golden["C"], pos=pos)
    return b, Fo


@pytest.mark.parametrize("hbond", [False, True])
@pytest.mark.parametrize("rcut", [10.0, -1.0])
def test_step_forces_vs_oracle(world, golden, rcut, hbond):
    try:
        for sizes, shapes in ((SMALL, (32, 0, 64, 128, 256)), (LARGE, (0, 64, 128, 256, 512))):
            b, Fo = batch(world, golden, sizes, rcut, hbond)
            for T in shapes:
                if T == 32:
                    for c in (0, 1):
                        assert world.lib.mmff_set_tuning(c, 0, 1, 32, 1) == 0
                else:
                    world.set_launch(T, 0)
                compare(b, step_forces(world, b), Fo)
                world.set_launch(0, 0)
                for c in (0, 1):
                    world.lib.mmff_set_tuning(c, -1, 1, 0, 0)
    finally:
        world.set_launch(0, 0)
        for c in (0, 1):
            world.lib.mmff_set_tuning(c, -1, 1, 0, 0)


def test_lists_off_and_wide_image_sets(world, golden):
    """Candidate rows (lists switched off; 24 images, more than the lists take)
    give the oracle's forces."""
    grid = grid_from_golden(golden)
    try:
        for npbc, lists in (((1, 1, 0), False), ((2, 2, 0), True)):
            b = S.make_systems([30, 60, 90, 130, 200], 19, topo_mode=1, sigma=0.05, npbc=npbc)
            world.set_params(flags=DEFAULT_FLAGS, npbc=npbc, Rcut=10.0)
            world.set_fire(FireParams())
            world.set_pair_lists(lists)
            world.grid_upload(golden["C"], grid)
            world.upload(b)
            pos = world.state()["pos"]
            Fo, _ = O.eval_forces(b, O.make_params(grid, flags=DEFAULT_FLAGS, npbc=npbc, Rcut=10.0), golden["C"], pos=pos)
            compare(b, step_forces(world, b), Fo)
    finally:
        world.set_pair_lists(True)
        world.set_params(flags=DEFAULT_FLAGS, Rcut=10.0)


@pytest.mark.parametrize("n", [700, 1000])
def test_largest_systems_still_relax(world, golden, n):
    """Systems near the shared-memory limit (velocities, topology or both in
    global memory): accepted with every forced block size that took them, and
    right."""
    grid = grid_from_golden(golden)
    b = S.make_systems([n], 23, topo_mode=1, sigma=0.0, cell=(200.0, 200.0, 40.0))
    world.set_params(flags=DEFAULT_FLAGS, npbc=(0, 0, 0), Rcut=-1.0)
    b.neighCell[:] = 0
    world.set_fire(FireParams())
    world.grid_upload(golden["C"], grid)
    world.upload(b)
    pos = world.state()["pos"]
    Fo, _ = O.eval_forces(b, O.make_params(grid, flags=DEFAULT_FLAGS, npbc=(0, 0, 0), Rcut=-1.0), golden["C"], pos=pos)
    try:
        for T in (0, 512):
            world.set_launch(T, 0)
            F = step_forces(world, b)
            err = np.abs(F - Fo).max() / np.abs(Fo).max()
            assert err < FTOL, err
            st = world.state()
            assert np.isfinite(st["vel"]).all()
    finally:
        world.set_launch(0, 0)
        world.set_params(flags=DEFAULT_FLAGS, Rcut=10.0)
