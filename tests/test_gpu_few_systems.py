"""Batches of few systems: relaxation by clusters of blocks (one system held by
2 to 8 of them, up to half as many systems as SMs) against one block per system,
and evaluation by a block per system against a warp each (more systems than SMs),
also with several size classes side by side."""
import numpy as np
import pytest

from conftest import grid_from_golden
from firecore_b200 import systems as S
from firecore_b200.world import DEFAULT_FLAGS, FireParams, World

pytestmark = pytest.mark.gpu
FTOL = 1e-5                      # forces: relative to the system's largest (the bar against the oracle)


@pytest.fixture(scope="module")
def world():
    return World(0)


def setup(w, golden, b, rcut):
    w.set_params(flags=DEFAULT_FLAGS, Rcut=rcut)
    w.set_fire(FireParams())
    w.grid_upload(golden["C"], grid_from_golden(golden))
    w.upload(b)


@pytest.mark.parametrize("rcut", [10.0, -1.0])
@pytest.mark.parametrize("nsys", [1, 19, 73, 74, 75])
def test_cluster_relaxation_is_block_relaxation(world, golden, nsys, rcut):
    """Ten steps: the paths differ by rounding, at most FTOL of a system's largest
    force each step, so its positions by FTOL Fmax (n dt)^2 / 2 undamped (twice
    that is allowed).  Then with a threshold between the systems' forces: the
    same ones retire at the first step."""
    sizes = [65, 66, 96, 100, 129, 200, 257, 350]
    b = S.make_systems([sizes[i % len(sizes)] for i in range(nsys)], 29, topo_mode=1, sigma=0.05)
    v = b.offsets()[2]
    n, dt = 10, FireParams().dt_max
    try:
        setup(world, golden, b, rcut)
        F, _ = world.eval(energy=False)
        pos, done = [], []
        for T in (0, 256):
            world.set_launch(T, 0)
            world.restore()
            world.relax(1, 0.0, conv_mode=1)
            fc = np.sort(world.state()["fconv"])
            gap = np.argmax(fc[1:] / fc[:-1]) if nsys > 1 else 0
            thr = np.sqrt(fc[gap] * fc[gap + 1]) if nsys > 1 else 2.0 * fc[0]
            world.restore()
            world.relax(n, thr, conv_mode=1)
            st = world.state()
            done.append((st["nsteps"] == 0, st["status"][st["nsteps"] == 0]))
            world.restore()
            world.relax(n, 0.0, conv_mode=1)
            st = world.state()
            pos.append(st["pos"])
        assert np.array_equal(done[0][0], done[1][0]) and np.array_equal(done[0][1], done[1][1])
        checked = 0
        for s in range(nsys):
            fmax = np.abs(F[v[s]:v[s + 1]]).max()
            if fmax > 1e3:               # atoms on top of an image: chaotic within these steps
                continue
            d = np.abs(pos[0][v[s]:v[s + 1]] - pos[1][v[s]:v[s + 1]]).max()
            assert d <= FTOL * fmax * (n * dt) ** 2, (int(b.natoms[s]), d, fmax)
            checked += 1
        assert checked >= 0.6 * nsys, checked
    finally:
        world.set_launch(0, 0)
        world.set_params(flags=DEFAULT_FLAGS, Rcut=10.0)


@pytest.mark.parametrize("rcut", [10.0, -1.0])
@pytest.mark.parametrize("sizes", [(32,), (20, 24, 33, 64), (24, 64, 65, 130, 300)])
def test_small_batch_evaluation_matches_large_batch(world, golden, sizes, rcut):
    b = S.make_systems(list(sizes), 31, topo_mode=1, sigma=0.05)
    rep = 160 // len(sizes) + 1
    try:
        setup(world, golden, b, rcut)
        few, Ef = world.eval()
        big = b.subset(list(range(b.nsys)) * rep)
        world.upload(big)
        many, Em = world.eval()
        v, vb = b.offsets()[2], big.offsets()[2]
        for s in range(big.nsys):
            r = s % b.nsys
            f, g = few[v[r]:v[r + 1]], many[vb[s]:vb[s + 1]]
            assert np.abs(f - g).max() <= FTOL * np.abs(f).max(), (s, np.abs(f - g).max())
            e = np.abs(Ef[r] - Em[s])
            assert np.all(e <= 1e-6 * np.abs(Ef[r]) + 1e-5), (s, e)
    finally:
        world.set_params(flags=DEFAULT_FLAGS, Rcut=10.0)
