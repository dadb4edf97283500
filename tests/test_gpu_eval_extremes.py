"""The force measure that evaluations leave: state's fconv after an evaluation is the
largest force norm of the system."""
import numpy as np
import pytest

from conftest import grid_from_golden
from firecore_b200 import systems as S
from firecore_b200.world import DEFAULT_FLAGS, World

pytestmark = pytest.mark.gpu
SIZES = [24, 32, 50, 64, 65, 130, 300]


@pytest.fixture(scope="module")
def world():
    return World(0)


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
