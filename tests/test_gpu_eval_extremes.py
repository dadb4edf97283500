"""Evaluations where fixed-point pair sums do not reach, and the force measure they leave.

Atoms on top of one another: forces of 10^8 eV/A and more, beyond the 2^20 that a term of
the sums holds; every launch shape returns them, at the bar of ordinary forces (1e-5 of the
largest), and a system whose other atoms are apart keeps its forces too.  State's fconv
after an evaluation is the largest force norm of the system."""
import numpy as np
import pytest

from conftest import grid_from_golden
from firecore_b200 import systems as S
from firecore_b200.world import DEFAULT_FLAGS, FireParams, World
from oracle import oracle as O

pytestmark = pytest.mark.gpu
SIZES = [24, 32, 50, 64, 65, 130, 300]


@pytest.fixture(scope="module")
def world():
    return World(0)


def close_pairs(b):
    """Two atoms of every molecule, not bonded nor ends of an angle, 0.4 A apart."""
    a, _, v = b.offsets()
    for s in range(b.nsys):
        n = int(b.natoms[s])
        ng = [set(int(x) for x in r if x >= 0) for r in b.neighs[a[s]:a[s] + n]]
        for i in range(n):
            for x in ng[i]:
                ng[x].add(i)
        i = 0
        near = ng[i] | set().union(*(ng[x] for x in ng[i])) | {i}
        j = next(x for x in range(n - 1, 0, -1) if x not in near)
        b.pos[v[s] + j] = b.pos[v[s] + i] + [0.3, 0.2, 0.17]
    return b


@pytest.mark.parametrize("rcut", [10.0, -1.0])
@pytest.mark.parametrize("copies", [1, 60])
def test_forces_of_overlapping_atoms(world, golden, rcut, copies):
    grid = grid_from_golden(golden)
    b = close_pairs(S.make_systems(SIZES, 53, topo_mode=1, sigma=0.05))
    try:
        world.set_params(flags=DEFAULT_FLAGS, Rcut=rcut)
        world.set_fire(FireParams())
        world.grid_upload(golden["C"], grid)
        world.upload(b.subset(list(range(b.nsys)) * copies))
        F, _ = world.eval()
        Fo, _ = O.eval_forces(b, O.make_params(grid, flags=DEFAULT_FLAGS, Rcut=rcut), golden["C"],
                              pos=world.state()["pos"][:len(b.pos)])
        fconv = world.state()["fconv"]
        v = b.offsets()[2]
        for s in range(b.nsys):
            f, ref = F[v[s]:v[s + 1]], Fo[v[s]:v[s + 1]]
            assert np.abs(ref).max() > 1e7
            assert np.abs(f - ref).max() <= 1e-5 * np.abs(ref).max(), (int(b.natoms[s]), np.abs(f).max(), np.abs(ref).max())
            # the measure: the largest norm, FP32
            assert abs(fconv[s] - np.linalg.norm(f, axis=1).max()) <= 1e-6 * fconv[s], (int(b.natoms[s]), fconv[s])
    finally:
        world.set_params(flags=DEFAULT_FLAGS, Rcut=10.0)


@pytest.mark.parametrize("copies,threads", [(1, 0), (60, 0), (1, 64), (1, 512)])
@pytest.mark.parametrize("energy", [True, False])
def test_measure_after_evaluation(world, golden, copies, threads, energy):
    b = S.make_systems(SIZES, 59, topo_mode=1, sigma=0.05)
    try:
        world.set_params(flags=DEFAULT_FLAGS, Rcut=10.0)
        world.grid_upload(golden["C"], grid_from_golden(golden))
        big = b.subset(list(range(b.nsys)) * copies)
        world.upload(big)
        world.set_launch(threads, 0)
        F = world.eval(energy)[0]
        fconv, v = world.state()["fconv"], big.offsets()[2]
        want = np.array([np.linalg.norm(F[v[s]:v[s + 1]], axis=1).max() for s in range(big.nsys)])
        assert np.abs(fconv - want).max() <= 1e-6 * want.max(), np.abs(fconv - want).max()
    finally:
        world.set_launch(0, 0)
