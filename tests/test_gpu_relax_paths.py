"""Relaxations and Langevin runs take the path they took before: end positions equal,
bit for bit, those stored in golden/relax_paths.npz (made by make_relax_golden.py there),
whatever shares the work -- a block per system, a cluster of blocks, more threads.

A path of some hundred steps amplifies the last bit of a force to 0.01 A and more in
single molecules, so there is no tolerance for another order of the sums; equal bits
it is.  Sizes: both forms of the small systems' pair sums, the edges of tiles and size
classes, with a cutoff (pair lists) and without (image rows), with and without
hydrogen bonds."""
import ctypes
import os
import sys

import numpy as np
import pytest

from conftest import grid_from_golden
from firecore_b200 import systems as S
from firecore_b200.world import DEFAULT_FLAGS, FireParams, World
from oracle import oracle as O

sys.path.insert(0, os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden"))
import make_relax_golden as M  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def world():
    return World(0)


@pytest.fixture(scope="module")
def paths():
    return dict(np.load(os.path.join(os.path.dirname(M.__file__), "relax_paths.npz")))


# clusters, a block each, more systems than SMs, blocks of several systems
@pytest.mark.parametrize("rcut,hbond,copies", [c + (n,) for c in M.CASES for n in (1, 5, 11)] + [(10.0, False, 600)])
def test_relaxation_path(world, golden, paths, rcut, hbond, copies):
    b = M.batch(hbond)
    ref = paths["pos_%g_%d" % (rcut, hbond)]
    try:
        M.setup(world, golden["C"], grid_from_golden(golden), b.subset(list(range(b.nsys)) * copies), rcut)
        pos = M.relaxed(world, hbond).reshape(copies, *ref.shape)
        v = b.offsets()[2]
        for s in range(b.nsys):
            got = pos[:, v[s]:v[s + 1]]
            assert np.array_equal(got, np.broadcast_to(ref[v[s]:v[s + 1]], got.shape), equal_nan=True), (
                int(b.natoms[s]), np.abs(got - ref[v[s]:v[s + 1]]).max())
        if not hbond:                                # the random stream goes by the vector's index in the batch
            assert np.array_equal(M.sampled(world)[:len(ref)], paths["md_%g" % rcut], equal_nan=True)
    finally:
        world.set_params(flags=DEFAULT_FLAGS, Rcut=10.0)


@pytest.mark.parametrize("n,rcut", [(850, -1.0), (1000, -1.0), (850, 10.0)])
def test_largest_systems_with_images(world, golden, n, rcut):
    """Near the shared-memory limit with shifted images: image rows whose sums and arrays
    are no longer in shared memory, pair lists; one step's forces against the FP64 oracle."""
    grid = grid_from_golden(golden)
    b = S.make_systems([n], 23, topo_mode=1, sigma=0.0, cell=(60.0, 60.0, 40.0))
    try:
        world.set_params(flags=DEFAULT_FLAGS, npbc=(1, 1, 0), Rcut=rcut)
        world.set_fire(FireParams())
        world.grid_upload(golden["C"], grid)
        world.upload(b)
        Fo, _ = O.eval_forces(b, O.make_params(grid, flags=DEFAULT_FLAGS, npbc=(1, 1, 0), Rcut=rcut), golden["C"],
                              pos=world.state()["pos"])
        world.relax(1, 0.0, conv_mode=1)
        F = np.zeros_like(Fo)
        assert world.lib.mmff_get_forces(F.ctypes.data_as(ctypes.c_void_p)) == 0
        err = np.abs(F - Fo).max() / np.abs(Fo).max()
        assert err < 1e-5, err                       # the bar of the evaluation
    finally:
        world.set_params(flags=DEFAULT_FLAGS, Rcut=10.0)
