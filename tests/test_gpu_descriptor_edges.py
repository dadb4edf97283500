"""Neighbour selection of the descriptors where it can go wrong: fewer than 32
neighbours, exactly 32, one more, many, with many equal distances (atoms on a
cubic lattice, exact in FP32, so that the order by (r, image, j) decides), and
periodic images at the edge of the reach.  Against the FP64 oracle: at most 32
terms exp(-t^2 / 0.18) of FP32, each good to a few 1e-7 and a distance error of
3e-7 A times the largest slope (2.0 per A): below 1e-4 in sum."""
import numpy as np
import pytest

from conftest import grid_from_golden
from firecore_b200 import learned as L
from firecore_b200 import systems as S
from firecore_b200.world import DEFAULT_FLAGS, World
from oracle import mlp_oracle as M

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def world():
    return World(0)


def lattice(shape, a):
    """Whole lattices: their centroid, the origin of the device's coordinates, is exact too."""
    g = np.stack(np.meshgrid(*[np.arange(k) for k in shape], indexing="ij"), -1).reshape(-1, 3)
    return g * a + np.array([1.0, 1.0, 4.0])


@pytest.mark.parametrize("edge", [7.0, 9.0, 11.0, 24.0])
def test_selection_on_a_lattice(world, golden, edge):
    cases = [((2, 2, 5), 1.0), ((2, 4, 4), 1.0), ((1, 3, 11), 0.5), ((1, 2, 17), 0.5), ((2, 3, 11), 1.0), ((5, 5, 5), 1.5)]
    b = S.make_systems([int(np.prod(c[0])) for c in cases], 37, topo_mode=1, sigma=0.0, cell=(edge, edge, 40.0))
    v = b.offsets()[2]
    rng = np.random.default_rng(5)
    for s, c in enumerate(cases):
        p = lattice(*c)
        b.pos[v[s]:v[s] + len(p)] = p[rng.permutation(len(p))]
    b.elements[:] = rng.integers(0, 4, len(b.elements))
    try:
        world.set_params(flags=DEFAULT_FLAGS, Rcut=10.0)
        world.grid_upload(golden["C"], grid_from_golden(golden))
        world.upload(b)
        prop = L.Proposal()
        prop.set_elements(b.elements)
        f = prop.features(int(b.natoms.sum()), z_top=0.0)
        pos = L.atom_rows(b, world.state()["pos"])
        fo = M.descriptors(pos, b.elements, b.natoms, b.lvec, (1, 1, 0), 0.0, np.zeros((len(pos), 3)))
        assert np.abs(f[:, :65] - fo[:, :65]).max() < 1e-4, np.abs(f[:, :65] - fo[:, :65]).max()
    finally:
        world.set_params(flags=DEFAULT_FLAGS, Rcut=10.0)
