"""relax_paths.npz: end positions of short relaxations, as the relaxation kernels of
commit 4f52328 gave them on a B200 (needs a GPU; run from the repository's root).

A relaxation amplifies the last bit of a force, so that another order of the same
sums ends elsewhere.  tests/test_gpu_relax_paths.py compares bits."""
import os
import sys

import numpy as np

sys.path.insert(0, os.getcwd())
from firecore_b200 import systems as S  # noqa: E402
from firecore_b200.world import DEFAULT_FLAGS, FireParams, World  # noqa: E402

SIZES = [20, 24, 31, 32, 33, 47, 60, 64, 65, 96, 128, 129, 200, 257, 330]
CASES = [(rcut, hbond) for rcut in (10.0, -1.0) for hbond in (False, True)]
STEPS = 200                     # 40 with hydrogen bonds
MD_STEPS = 40


def batch(hbond):
    return S.make_systems(SIZES, 41, topo_mode=1, sigma=0.15, rotate=True, hbond=hbond)


def setup(w, coefs, grid, b, rcut):
    w.set_params(flags=DEFAULT_FLAGS, npbc=(1, 1, 0), Rcut=rcut)
    w.set_fire(FireParams())
    w.grid_upload(coefs, grid)
    w.upload(b)


def relaxed(w, hbond):
    w.restore()
    w.relax(40 if hbond else STEPS, 1e-4, conv_mode=1)
    return w.state()["pos"]


def sampled(w):
    w.restore()
    w.set_md(dt=0.05, gamma=0.1, T=300.0, seed=5)
    w.md(MD_STEPS)
    return w.state()["pos"]


if __name__ == "__main__":
    here = os.path.dirname(os.path.abspath(__file__))
    sys.path.insert(0, os.path.dirname(here))
    from conftest import grid_from_golden
    g = dict(np.load(os.path.join(here, "mmff_small.npz")))
    w, out = World(0), {}
    for rcut, hbond in CASES:
        setup(w, g["C"], grid_from_golden(g), batch(hbond), rcut)
        out["pos_%g_%d" % (rcut, hbond)] = relaxed(w, hbond)
        if not hbond:
            out["md_%g" % rcut] = sampled(w)
    np.savez_compressed(sys.argv[1] if len(sys.argv) > 1 else os.path.join(here, "relax_paths.npz"), **out)
