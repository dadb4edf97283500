"""Relaxations and Langevin runs take the path they took before: end positions equal,
bit for bit, those stored in golden/relax_paths.npz (made by make_relax_golden.py there),
whatever shares the work -- a block per system, a cluster of blocks, more threads.

A path of some hundred steps amplifies the last bit of a force to 0.01 A and more in
single molecules, so there is no tolerance for another order of the sums; equal bits
it is.  Sizes: both forms of the small systems' pair sums, the edges of tiles and size
classes, with a cutoff (pair lists) and without (image rows), with and without
hydrogen bonds."""
import os
import sys

import numpy as np
import pytest

from conftest import grid_from_golden
from firecore_b200.world import DEFAULT_FLAGS, World

sys.path.insert(0, os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden"))
import make_relax_golden as M  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def world():
    return World(0)


@pytest.fixture(scope="module")
def paths():
    return dict(np.load(os.path.join(os.path.dirname(M.__file__), "relax_paths.npz")))


@pytest.mark.parametrize("rcut,hbond", M.CASES)
@pytest.mark.parametrize("copies", [1, 5, 11])      # clusters, a block each, more systems than SMs
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
