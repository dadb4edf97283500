"""Grid build with many Coulomb images (the far ones interpolated) against the
direct FP64 sum over every image and an FFT / dense spline solve.

Bound: the interpolation leaves less than e^-40 per source, so what remains is
the rounding of FP64 sums of n terms of alternating sign.  Their absolute sum
is S = k_e sum_j |Q_j| sum_images 1/r; sums in another order differ by a few
eps * S (random-walk rounding), taken as 64 eps S here, and the spline solve
amplifies node errors by at most 3 per axis (largest entry sum of the inverse
of (1 4 1)/6 is 3): 27 * 64 eps S.
"""
import numpy as np
import pytest

from firecore_b200 import systems as S
from firecore_b200.world import World

pytestmark = pytest.mark.gpu
KE = 14.3996448915


def reference(sub):
    import torch
    dev, f8 = "cuda", torch.float64
    g = sub.grid
    ax = [torch.arange(g.n[k], device=dev, dtype=f8) * g.step[k] + g.pos0[k] for k in range(3)]
    V = torch.zeros(*g.n, 3, device=dev, dtype=f8)
    A = torch.zeros(*g.n, device=dev, dtype=f8)
    lv = np.asarray(sub.lvec)

    def cells(n):
        return [lv[0] * i + lv[1] * j + lv[2] * k for k in range(-n[2], n[2] + 1) for j in range(-n[1], n[1] + 1)
                for i in range(-n[0], n[0] + 1)]
    for p, (R0, E0, Q, _) in zip(sub.spos, sub.sREQ):
        def r2(sh):
            x, y, z = (float(p[c] - sh[c]) for c in range(3))
            return ((ax[0] - x) ** 2)[:, None, None] + ((ax[1] - y) ** 2)[None, :, None] + ((ax[2] - z) ** 2)[None, None, :]
        for sh in cells(sub.nPBC_mors):
            e = torch.exp(-sub.alphaMorse * (torch.sqrt(r2(sh)) - R0))
            V[..., 0] += E0 * e * e
            V[..., 1] -= 2.0 * E0 * e
        s = torch.zeros(*g.n, device=dev, dtype=f8)
        for sh in cells(sub.nPBC_coul):
            s += torch.rsqrt(r2(sh))
        V[..., 2] += KE * Q * s
        A += KE * abs(Q) * s
    nx, ny, nz = g.n
    lam = [(4 + 2 * torch.cos(2 * np.pi * torch.arange(n, device=dev, dtype=f8) / n)) / 6 for n in (nx, ny)]
    C = torch.fft.ifft2(torch.fft.fft2(V, dim=(0, 1)) / (lam[0][:, None] * lam[1][None])[:, :, None, None], dim=(0, 1)).real
    M = (torch.diag(torch.full((nz,), 4.0)) + torch.diag(torch.ones(nz - 1), 1) + torch.diag(torch.ones(nz - 1), -1)).to(C) / 6
    C = torch.linalg.solve(M, C.permute(2, 0, 1, 3).reshape(nz, -1)).reshape(nz, nx, ny, 3).permute(1, 2, 0, 3)
    return C.cpu().numpy(), float(A.max()), V.abs().amax((0, 1, 2)).cpu().numpy()


# the cell's own box (odd node counts, not multiples of the nodes a thread takes);
# a box that is not the cell's, off its corner; few images (direct sum); a skewed
# cell; a box larger than the cell (every image direct); a long z axis
CASES = {
    "cell": dict(step=0.25, nz=33, images=(9, 7, 0)),
    "shifted": dict(step=0.23, nz=24, images=(8, 8, 0), pos0=(3.1, -4.2, 2.0), n=(37, 42, 24)),
    "few": dict(step=0.4, nz=17, images=(1, 1, 0)),
    "skewed": dict(step=0.25, nz=20, images=(6, 6, 0), skew=3.3),
    "wide": dict(step=0.5, nz=12, images=(4, 4, 0), n=(61, 59, 12)),
    "stacked": dict(step=0.3, nz=40, images=(4, 4, 2)),
    "long": dict(step=1.1, nz=5000, images=(1, 1, 0), z=0.01),
}


@pytest.mark.parametrize("name", list(CASES))
def test_grid_build_many_images_vs_direct_sum(name):
    c = CASES[name]
    sub = S.make_slab(ncell=2, layers=2, grid_step=c["step"], nz=c["nz"], nPBC_coul=c["images"])
    rng = np.random.default_rng(3)
    sub.spos = sub.spos + rng.normal(0, 0.05, sub.spos.shape)
    g = sub.grid
    sub.grid = S.GridSpec(tuple(c.get("n", g.n)), tuple(c.get("pos0", g.pos0)),
                          (g.step[0], g.step[1], c.get("z", g.step[2])))
    if "skew" in c:
        sub.lvec = np.array(sub.lvec, float)
        sub.lvec[1, 0] += c["skew"]
    C = World(0).grid_build(sub, return_coefs=True)
    ref, asum, vmax = reference(sub)
    eps = np.finfo(float).eps
    for k, s in enumerate((vmax[0], vmax[1], asum)):      # Morse sums have one sign: their maximum bounds them
        err = np.abs(C[..., k] - ref[..., k]).max()
        assert err <= 27 * 64 * eps * s, (name, k, err, 27 * 64 * eps * s)
