"""Performance cases of the B200 multi-system MMFF relaxer.

What a program does with this package: it types or generates a set of molecules,
uploads them once (topology and force-field parameters: the plan it keeps), and
then evaluates or relaxes them again and again from new start geometries,
samples them with the Langevin drive, moves them with the learned proposal,
trains that proposal, screens sets of new molecules, and builds the substrate
grid.  Every case goes through the public classes ``World`` and ``Proposal``
with host arrays in and host arrays out, as INTEGRATION's examples do.

Geometries and training rows come from the seed; the topology of a case is
fixed by the case itself.  Molecules, slab and grid are the ones of
``firecore_b200.systems``: C:N:O:H = 10:2:2:10 trees of 20-400 atoms on a
rock-salt slab, GridFF 226 x 226 x 200, 10 A cutoff, FIRE with a 10 eV/A clamp.
"""
import math

import numpy as np
import torch

from firecore_b200 import learned as L
from firecore_b200 import systems as S
from firecore_b200.world import DEFAULT_FLAGS, FireParams, World

KE = 14.3996448915           # eV A / e^2
CELL = 22.56                 # edge of the periodic cell, 4 x 5.64 A
NBATCH_TILES = 512           # 65536 atoms per training batch
_DEV = "cuda"


def _t(a, dt=torch.float64):
    return torch.as_tensor(np.ascontiguousarray(a), device=_DEV).to(dt)


# ------------------------------------------------------------------ the cases

def listed():
    return [
        # one small molecule's replicas, all pairs x 9 images, as a FireCore script evaluates them: latency
        dict(name="eval_16x24", kind="eval", nsys=16, lo=24, hi=24, same=True, rcut=-1.0, topo=3),
        # one energy-and-force evaluation of a mixed batch
        dict(name="eval_uneven_2048", kind="eval", nsys=2048, lo=20, hi=400, same=False, rcut=10.0, topo=11),
        # the reference's CPU-runnable configuration: 16 replicas, no cutoff, sum f^2 < Fconv^2, <= 2000 steps
        dict(name="relax_16x24", kind="relax", nsys=16, lo=24, hi=24, same=True, rcut=-1.0, flim=-1.0, steps=2000,
             mode=0, tuned=False, topo=3),
        # replicas of one 60-atom molecule at GPU scale, launch shapes as the library chooses them
        dict(name="relax_4096x60", kind="relax", nsys=4096, lo=60, hi=60, same=True, rcut=10.0, flim=10.0, steps=2000,
             mode=1, tuned=False, topo=1),
        # the production queue: uneven molecules, autotuned launch shapes, one graph per relaxation
        dict(name="relax_uneven_3000", kind="relax", nsys=3000, lo=20, hi=400, same=False, rcut=10.0, flim=10.0,
             steps=2000, mode=1, tuned=True, topo=2),
        # a few large molecules: fewer systems than the chip has SMs
        dict(name="relax_37_large", kind="relax", nsys=37, lo=301, hi=397, same=False, rcut=10.0, flim=10.0, steps=400,
             mode=1, tuned=False, topo=5),
        # FireCore's own semantics (no cutoff: all pairs x 9 images) on mixed molecules
        dict(name="relax_allpairs_300", kind="relax", nsys=300, lo=20, hi=400, same=False, rcut=-1.0, flim=10.0,
             steps=300, mode=0, tuned=False, topo=7),
        # Langevin sampling of an odd-sized molecule
        dict(name="md_1000x37", kind="md", nsys=1000, lo=37, hi=37, same=True, rcut=10.0, flim=10.0, steps=300, topo=9),
        # screening: new molecules every call, uploaded, relaxed for a while, read back
        dict(name="screen_333", kind="screen", nsys=333, lo=20, hi=150, same=False, rcut=10.0, flim=10.0, steps=200,
             mode=1, topo=13),
        # two energy-gated learned moves of a mixed batch
        dict(name="learned_moves_2048", kind="warm", nsys=2048, lo=20, hi=400, same=False, rcut=10.0, topo=11),
        # training of the proposal: 200 AdamW steps of 65536 atoms over a ragged training set
        dict(name="train_107001", kind="train", rows=107001, steps=200, tiles=NBATCH_TILES),
        # substrate grid: direct sums over 51 x 51 images and the spline fit, 0.25 A spacing
        dict(name="grid_0.25A", kind="grid", ncell=4, layers=3, step=0.25, nz=80, images=25),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["eval", "relax", "relax", "relax", "relax", "md", "screen", "warm", "train", "grid"])
    topo = rng.randrange(100, 1 << 20)
    if kind == "train":
        return dict(kind=kind, rows=_log(rng, 500, 107000), steps=rng.randrange(20, 200), tiles=rng.randrange(8, 512))
    if kind == "grid":
        return dict(kind=kind, ncell=rng.choice([2, 3, 4]), layers=rng.choice([2, 3]), step=rng.uniform(0.25, 0.4),
                    nz=rng.randrange(40, 80), images=rng.randrange(4, 25))
    lo = _log(rng, 20, 250)
    same = rng.random() < 0.4
    hi = lo if same else min(400, int(lo * rng.uniform(1.1, 6.0)))
    c = dict(kind=kind, lo=lo, hi=hi, same=same, topo=topo)
    # atoms in the batch: no more than the largest listed case holds
    most = {"eval": 2048 * 127, "relax": 3000 * 127, "md": 1000 * 37, "screen": 333 * 65, "warm": 2048 * 127}[kind]
    top = max(12, int(most / (0.5 * (lo + hi))))
    c["nsys"] = _log(rng, 1 if kind != "warm" else 512, min(top, 4096))
    c["rcut"] = 10.0 if kind in ("warm", "md") or rng.random() < 0.75 else -1.0
    if kind in ("relax", "md", "screen"):
        c["flim"] = 10.0
        c["steps"] = _log(rng, 50, {"relax": 1000, "md": 300, "screen": 200}[kind])
    if kind in ("relax", "screen"):
        c["mode"] = rng.choice([0, 1])
    if kind == "relax":
        c["tuned"] = rng.random() < 0.3 and c["nsys"] >= 256
        if c["rcut"] < 0:
            c["nsys"] = min(c["nsys"], max(8, int(300 * 127 / (0.5 * (lo + hi)))))
            c["steps"] = min(c["steps"], 300)
    return c


# ------------------------------------------------------------------ inputs

_world = None
_plan = {"systems": None, "grid": None}       # what the device world holds now
_kept = {}                                     # batches by case, the slab's grid


def _w():
    global _world
    if _world is None:
        _world = World(0)
    return _world


def _slab():
    return S.make_slab(nPBC_coul=(4, 4, 0))


def _sizes(case, topo):
    if case["same"]:
        return np.full(case["nsys"], case["lo"], np.int32)
    return S.loguniform_sizes(case["nsys"], topo, case["lo"], case["hi"])


def _molecules(case, topo):
    return S.make_systems(_sizes(case, topo), topo, topo_mode=0 if case["same"] else 1, sigma=0.0, rotate=True)


def _key(case):
    return tuple(sorted((k, v) for k, v in case.items() if k != "name"))


def _base(case):
    """The case's molecules (topology, parameters, a geometry without noise)."""
    key = _key(case)
    if _kept.get("key") != key:
        b = _molecules(case, case["topo"])
        if case["kind"] in ("eval", "warm"):
            b = _apart(b)
        sysi = np.repeat(np.arange(b.nsys), b.nvecs)
        inside = np.arange(int(b.nvecs.sum())) - np.repeat(b.offsets()[2][:-1], b.nvecs)
        _kept.update(key=key, batch=b, sys=sysi, atom=inside < np.repeat(b.natoms, b.nvecs))
    return _kept


def _chunks(b, most=6_000_000):
    """Systems of like size, a few million atom pairs at a time: (systems, atom there?, vector rows, atom rows)."""
    a0, _, v0 = b.offsets()
    order = np.argsort(b.natoms, kind="stable")
    p = 0
    while p < len(order):
        q = p + 1
        while q < len(order) and (q - p + 1) * int(b.natoms[order[q]]) ** 2 <= most:
            q += 1
        ss = order[p:q]
        p = q
        k = np.arange(int(b.natoms[ss].max()))
        has = k[None] < b.natoms[ss][:, None]
        yield ss, has, np.where(has, v0[ss][:, None] + k, 0), np.where(has, a0[ss][:, None] + k, 0)


def _apart(b):
    """Molecules with atoms that overlap pushed apart (to 2 A, periodic images too; bonded ones excepted), those
    where that fails replaced by one of like size: an evaluation, and the learned moves' energy gate, see molecules
    and not the 10^6 eV/A of two random branches through one another."""
    pos, near = b.pos.copy(), np.zeros(b.nsys)
    for ss, has, vi, ai in _chunks(b):
        x, live = _t(pos[vi]), torch.as_tensor(has, device=_DEV)
        ng = torch.as_tensor(np.where(has[..., None], b.neighs[ai], -1).astype(np.int64), device=_DEV)
        N = has.shape[1]
        off = ~(live[:, :, None] & live[:, None, :]) | torch.eye(N, dtype=torch.bool, device=_DEV)
        for c in range(4):
            m = torch.zeros_like(off)
            m.scatter_(2, ng[:, :, c].clamp_min(0)[..., None], (ng[:, :, c] >= 0)[..., None])
            off |= m | m.transpose(1, 2)
        for _ in range(40):
            d = x[:, :, None, :] - x[:, None, :, :]
            d[..., :2] -= CELL * torch.round(d[..., :2] / CELL)
            r = torch.sqrt((d * d).sum(-1) + 1e-6)
            push = torch.where(off | (r > 2.0), torch.zeros_like(r), (2.0 - r) / r)
            x = x + 0.25 * (d * push[..., None]).sum(2)
        near[ss] = torch.where(off, torch.full_like(r, 9.0), r).amin((1, 2)).cpu().numpy()
        pos[vi[has]] = x[live].cpu().numpy()
    b.pos = pos
    good = np.flatnonzero(near > 1.6)
    good = good[np.argsort(b.natoms[good], kind="stable")]
    at = np.searchsorted(b.natoms[good], b.natoms).clip(0, len(good) - 1)
    return b.subset(np.where(near > 1.6, np.arange(b.nsys), good[at]))


def _geometry(k, seed, noise):
    """New start geometry of the kept molecules: turned about the surface normal, shifted along the surface, noise."""
    b, sysi, atom = k["batch"], k["sys"], k["atom"]
    rng = np.random.default_rng([17, seed])
    phi = rng.uniform(0, 2 * np.pi, b.nsys)
    if noise < 0.1:          # the square cell's own turns: a molecule stays clear of its images
        phi = np.round(phi / (np.pi / 2)) * (np.pi / 2)
    shift = rng.uniform(-0.5, 0.5, (b.nsys, 2)) * 5.64
    n = atom.astype(np.float64)
    cnt = np.bincount(sysi, n, b.nsys)
    cen = np.stack([np.bincount(sysi, n * b.pos[:, c], b.nsys) / cnt for c in (0, 1)], 1)
    c, s = np.cos(phi)[sysi], np.sin(phi)[sysi]
    u = b.pos[:, :2] - np.where(atom[:, None], cen[sysi], 0.0)
    pos = b.pos.copy()
    pos[:, 0], pos[:, 1] = c * u[:, 0] - s * u[:, 1], s * u[:, 0] + c * u[:, 1]
    pos[atom, :2] += (cen + shift)[sysi[atom]]
    pos[atom] += rng.normal(0, noise, (int(atom.sum()), 3))
    return pos


def _noise(case):
    return 0.05 if case["kind"] in ("eval", "warm") else 0.15


def _load_grid(w):
    if _plan["grid"] != "slab":
        w.grid_build(_slab())
        _plan["grid"], _plan["systems"] = "slab", None


def _forces(w, case):
    w.set_params(flags=DEFAULT_FLAGS, npbc=(1, 1, 0), Rcut=case["rcut"])
    w.set_fire(FireParams(Flim=case.get("flim", -1.0)))


def _load(case):
    """The plan: force-field switches, systems on the device, launch shapes, the network."""
    key = _key(case)
    w = _w()
    if _plan["systems"] == key and _plan["grid"] == "slab":
        return w
    _load_grid(w)
    _forces(w, case)
    w.set_graph(bool(case.get("tuned")))
    for c in range(6):
        w.lib.mmff_set_tuning(c, -1, 1, 0, 0)
    b = _base(case)["batch"]
    w.upload(b)
    if case.get("tuned"):
        w.autotune(nstep_probe=20)
    if case["kind"] == "warm":
        k = _kept
        prop = L.Proposal()
        p = L.init_params(4)
        p["W3"][:3] *= 4.0
        prop.set_params(p, _FMEAN, _FSTD, 0.2)
        prop.set_elements(b.elements)
        prop.set_projection(1)
        k["prop"] = prop
    _plan["systems"] = key
    return w


# feature statistics of the generated molecules (radial bins per element channel, height, grid force)
_FMEAN = np.concatenate([np.full(64, 0.9), [9.0, 0.0, 0.0, 0.0]]).astype(np.float32)
_FSTD = np.concatenate([np.full(64, 1.1), [6.0, 0.3, 0.3, 0.6]]).astype(np.float32)


def _rows(case, seed):
    """Training rows like the descriptors': non-negative radial bins, a height, a force; targets a smooth function of them."""
    g = torch.Generator().manual_seed(1000 + seed)
    n = case["rows"]
    F = torch.randn(n, 68, generator=g)
    F[:, :64] = (F[:, :64] * 1.1 + 0.9).clamp_min_(0)
    F[:, 64] = F[:, 64].abs() * 6 + 3
    F[:, 65:] *= 0.3
    T = 0.15 * torch.tanh(F[:, 65:68] * 3) + 0.03 * (F[:, 0:3] - F[:, 16:19]) + 0.05 * torch.randn(n, 3, generator=g)
    return F.numpy(), T.numpy()


def _train_start():
    p = L.init_params(2)
    p["W3"][:3] *= 10.0
    return p


def prepare(case, seed):
    kind = case["kind"]
    if kind == "grid":
        rng = np.random.default_rng([23, seed])
        sub = S.make_slab(ncell=case["ncell"], layers=case["layers"], grid_step=case["step"], nz=case["nz"],
                          nPBC_coul=(case["images"], case["images"], 0))
        sub.spos = sub.spos + rng.normal(0, 0.03, sub.spos.shape)      # a relaxed, slightly rumpled slab
        return dict(case=case, sub=sub, w=_w())
    if kind == "train":
        F, T = _rows(case, seed)
        _w()
        return dict(case=case, F=F, T=T, p=_train_start(), prop=L.Proposal())
    if kind == "screen":
        w = _w()
        _load_grid(w)
        _forces(w, case)
        w.set_graph(False)
        for c in range(6):
            w.lib.mmff_set_tuning(c, -1, 1, 0, 0)
        _plan["systems"] = None
        b = S.make_systems(_sizes(case, case["topo"]), 7919 * seed + case["topo"], topo_mode=1, sigma=0.15,
                           rotate=True)
        return dict(case=case, w=w, batch=b)
    w = _load(case)
    return dict(case=case, w=w, pos=_geometry(_base(case), seed, _noise(case)), prop=_kept.get("prop"))


# ------------------------------------------------------------------ one pass

def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "grid":
        _plan["grid"] = None
        return state["w"].grid_build(state["sub"], return_coefs=True)
    if kind == "train":
        prop = state["prop"]
        prop.set_params(state["p"], _FMEAN, _FSTD, 0.2)
        prop.set_data(state["F"], state["T"])
        losses = prop.train(case["steps"], batch_tiles=case["tiles"], lr=1e-3, wd=0.01)
        return dict(losses=losses, **prop.params())
    if kind == "screen":
        w = state["w"]
        _plan["systems"] = None
        w.upload(state["batch"])
        w.relax(case["steps"], 1e-4, conv_mode=case["mode"])
        return w.state()["pos"]
    w = _load(case)
    w.set_state(state["pos"], None, reset_fire=True)
    if kind == "eval":
        F, E = w.eval(energy=True)
        return dict(F=F, E=E)
    if kind == "relax":
        # step counts, status, velocities and FIRE scalars at the end hang on the last bits of the path that led
        # there: the geometry is the result
        w.relax(case["steps"], 1e-4, conv_mode=case["mode"])
        return w.state()["pos"]
    if kind == "md":
        w.set_md(dt=0.05, gamma=0.1, T=300.0, seed=5)
        w.md(case["steps"])
        s = w.state()
        return dict(pos=s["pos"], vel=s["vel"])
    # learned moves
    acc = state["prop"].warmstart(w.batch.nsys, nsteps=2)
    return dict(accepted=acc, pos=w.state()["pos"])


# ------------------------------------------------------------------ what a pass cannot do without

def _sums(case):
    """(atoms, nodes, ordered pair-images inside the cutoff) of the batch, from the sizes alone."""
    n = _sizes(case, case["topo"]).astype(np.float64)
    if case["rcut"] > 0:
        # share of a molecule's own pairs inside 10 A: all of them up to ~60 atoms, half at 400
        pairs = n * (n - 1) * np.minimum(1.0, (70.0 / n) ** 0.37)
    else:
        pairs = 9.0 * n * (n - 1)
    return n.sum(), 0.58 * n.sum(), pairs.sum()


def work(case):
    kind = case["kind"]
    if kind == "grid":
        ncell, nz = case["ncell"], case["nz"]
        nx = round(5.64 * ncell / case["step"])
        nodes = nx * nx * nz
        terms = 4 * ncell * ncell * case["layers"] * nodes
        # per image: 3 subtractions, 6 for r^2, a root, an addition; Morse over 9 images ~25 each; 3 line solves
        return {"bytes": nodes * 24.0, "flops": terms * (11.0 * (2 * case["images"] + 1) ** 2 + 9 * 25.0) + nodes * 3 * 3 * 6.0}
    if kind == "train":
        rows = min(case["tiles"] * 128, case["rows"])
        return {"bytes": case["rows"] * (68 + 3) * 4.0 + 28944 * 8.0, "flops": case["steps"] * rows * 152.8e3}
    na, nn, pairs = _sums(case)
    nv = na + nn
    # 32 per ordered pair-image, ~700 per node (bonds, angles, pi terms), 64 x 11 per grid sample, ~40 per vector
    step = 32.0 * pairs + 700.0 * nn + 64 * 11.0 * na + 40.0 * nv
    if kind == "eval":
        return {"bytes": nv * (12 + 24.0), "flops": step}
    if kind == "warm":
        return {"bytes": nv * (24 + 24.0), "flops": 9 * step + 2 * na * 51e3}
    # most systems run all steps, the others about two thirds of them
    steps = case["steps"] * (0.9 if case["steps"] > 1000 else 1.0)
    return {"bytes": nv * (24 + 24.0), "flops": steps * step}


def tolerance(case):
    """About four times the largest difference seen between launch shapes that sum in another order, pair lists on and
    off, and start positions moved by 3e-7 A (half a unit in the last place of the FP32 coordinates)."""
    kind = case["kind"]
    if kind == "eval":
        return {"rel": 1e-5, "max": 4e-4}
    if kind == "grid":       # FP64 sums of 10^6 alternating terms
        return {"rel": 1e-10, "max": 1e-9}
    if kind == "train":      # bf16 operands: rounding flips travel through 200 steps
        return {"rel": 4e-3, "max": 3e-2}
    if kind == "warm":       # a few molecules in a thousand sit at an energy tie of the gate
        return {"rel": 2e-4, "max": 1e-2, "differ": 0.01}
    if kind == "md":
        return {"rel": 0.02, "max": 0.99}
    # relaxations: the end points of the soft modes, and of molecules still moving at the step limit, spread; with a
    # cutoff (forces step there) far more than without
    if case["steps"] <= 300:
        return {"rel": 2e-4, "max": 2e-2}
    return {"rel": 0.02, "max": 0.99} if case["rcut"] > 0 else {"rel": 2e-3, "max": 5e-2}


# ------------------------------------------------------------------ 64 bits

def _node_potentials(sub):
    """Pauli, London and Coulomb node values [nx, ny, nz, 3]: direct sums over substrate atoms and images."""
    g = sub.grid
    ax = [torch.arange(g.n[k], device=_DEV, dtype=torch.float64) * g.step[k] + g.pos0[k] for k in range(3)]
    V = torch.zeros(*g.n, 3, device=_DEV, dtype=torch.float64)
    a = sub.alphaMorse
    L3 = np.asarray(sub.lvec, np.float64)

    def cells(npbc):
        return [L3[0] * ix + L3[1] * iy + L3[2] * iz for iz in range(-npbc[2], npbc[2] + 1)
                for iy in range(-npbc[1], npbc[1] + 1) for ix in range(-npbc[0], npbc[0] + 1)]
    cell2 = g.n[0] * g.n[1]
    for near, images in ((True, cells(sub.nPBC_mors)), (False, cells(sub.nPBC_coul))):
        images = np.array(images)
        for j in range(len(sub.spos)):
            R0, E0, Q = (float(sub.sREQ[j, c]) for c in range(3))
            z2 = (ax[2] - float(sub.spos[j, 2])) ** 2
            for p in range(0, len(images), 64):
                x, y = (_t(float(sub.spos[j, c]) - images[p:p + 64, c]) for c in (0, 1))
                xy = (((ax[0] - x[:, None]) ** 2)[:, :, None] + ((ax[1] - y[:, None]) ** 2)[:, None, :]).reshape(-1, cell2, 1)
                r2 = xy + z2
                if near:
                    e = torch.exp(-a * (torch.sqrt(r2) - R0))
                    V[..., 0] += E0 * (e * e).sum(0).reshape(g.n)
                    V[..., 1] += -2.0 * E0 * e.sum(0).reshape(g.n)
                else:
                    V[..., 2] += KE * Q * r2.rsqrt_().sum(0).reshape(g.n)
    return V


def _fit(V):
    """Cubic B-spline coefficients: (c[i-1] + 4 c[i] + c[i+1]) / 6 = v[i], periodic in x and y, zero outside in z."""
    nx, ny, nz = V.shape[:3]
    lam = [(4 + 2 * torch.cos(2 * math.pi * torch.arange(n, device=_DEV, dtype=torch.float64) / n)) / 6 for n in (nx, ny)]
    C = torch.fft.fft2(V, dim=(0, 1)) / (lam[0][:, None] * lam[1][None, :])[:, :, None, None]
    C = torch.fft.ifft2(C, dim=(0, 1)).real
    M = (torch.diag(torch.full((nz,), 4.0)) + torch.diag(torch.ones(nz - 1), 1) + torch.diag(torch.ones(nz - 1), -1)).to(C) / 6
    return torch.linalg.solve(M, C.permute(2, 0, 1, 3).reshape(nz, -1)).reshape(nz, nx, ny, 3).permute(1, 2, 0, 3)


def _grid_terms(sub, C, pos, REQ):
    """Forces [n, 3] and energies [n] of atoms in the spline grid."""
    g = sub.grid
    ea = torch.exp(sub.alphaMorse * REQ[:, 0])
    PLQ = torch.stack([ea * ea * REQ[:, 1], ea * REQ[:, 1], REQ[:, 2]], 1)
    u = (pos - _t(g.pos0)) / _t(g.step)
    fl = torch.floor(u)
    i0 = fl.long()
    t = u - fl
    i0[:, 2] = i0[:, 2].clamp(3, g.n[2] - 5)

    def basis(t):
        s = 1 - t
        b = torch.stack([s ** 3, 3 * t * t * (t - 2) + 4, 3 * t * (1 + t - t * t) + 1, t ** 3], 1) / 6
        d = torch.stack([-s * s, 3 * t * t - 4 * t, -3 * t * t + 2 * t + 1, t * t], 1) / 2
        return b, d
    B = [basis(t[:, k]) for k in range(3)]
    k4 = torch.arange(4, device=_DEV) - 1
    ix = (i0[:, 0:1] + k4) % g.n[0]
    iy = (i0[:, 1:2] + k4) % g.n[1]
    iz = i0[:, 2:3] + k4
    flat = (ix[:, :, None, None] * g.n[1] + iy[:, None, :, None]) * g.n[2] + iz[:, None, None, :]
    c = (C.reshape(-1, 3)[flat] * PLQ[:, None, None, None, :]).sum(-1)
    e = lambda x, y, z: torch.einsum("nabc,na,nb,nc->n", c, x, y, z)  # noqa: E731
    E = e(B[0][0], B[1][0], B[2][0])
    F = torch.stack([-e(B[0][1], B[1][0], B[2][0]) / g.step[0], -e(B[0][0], B[1][1], B[2][0]) / g.step[1],
                     -e(B[0][0], B[1][0], B[2][1]) / g.step[2]], 1)
    return F, E


def _ljqh(r2, R, E, Q, H):
    ir2 = 1 / r2
    u6 = (R * R * ir2) ** 3
    return u6 * E * (u6 - 2) + Q * torch.sqrt(ir2) + u6 * u6 * E * H


def _bonded_energy(b, pos, off):
    """Bonded energy per node: bonds, pi-pi, pi-sigma, angles, and minus the plain pair term of each angle's ends."""
    a0, n0, v0 = off
    sysn = np.repeat(np.arange(b.nsys), b.nnode)
    loc = np.arange(len(sysn)) - n0[sysn]
    at = torch.as_tensor(v0[sysn] + loc, device=_DEV)
    row = a0[sysn] + loc
    ng = b.neighs[row].astype(np.int64)
    valid = np.cumprod(ng >= 0, 1).astype(bool)
    natoms = b.natoms[sysn].astype(np.int64)
    ok = torch.as_tensor(valid, device=_DEV)
    nb = np.where(valid, ng, 0)
    nvec = torch.as_tensor(v0[sysn][:, None] + nb, device=_DEV)
    cell = b.neighCell[row].astype(np.int64)
    sh = np.stack([(cell % 3 - 1) * CELL, (cell // 3 % 3 - 1) * CELL, 0.0 * cell], -1)
    h = pos[nvec] + _t(np.where(valid[..., None], sh, 0.0)) - pos[at][:, None]
    h = torch.where(ok[..., None], h, torch.ones_like(h))
    l = h.norm(dim=-1)
    u = h / l[..., None]
    pi = pos[torch.as_tensor(v0[sysn] + natoms + loc, device=_DEV)]
    once = ok & torch.as_tensor(loc[:, None] < nb, device=_DEV)
    E = (0.5 * _t(b.bKs) * (l - _t(b.bLs)) ** 2 * once).sum(1)
    kpp = _t(b.Kpp)
    isnode = once & torch.as_tensor(nb < b.nnode[sysn][:, None], device=_DEV) & (kpp > 1e-6)
    pj = pos[torch.as_tensor(np.where(nb < b.nnode[sysn][:, None], (v0[sysn] + natoms)[:, None] + nb, 0), device=_DEV)]
    E = E + (kpp * (1 - (pi[:, None] * pj).sum(-1).abs()) * isnode).sum(1)
    ap, ksp = _t(b.apars), _t(b.Ksp)
    cps = (pi[:, None] * u).sum(-1) - ap[:, 3:4]
    E = E + (ksp * cps * cps * (ok & (ksp > 1e-6))).sum(1)
    R = _t(b.REQs)
    ra = torch.as_tensor(a0[sysn][:, None] + nb, device=_DEV)
    for i in range(3):
        for j in range(i + 1, 4):
            both = ok[:, i] & ok[:, j]
            c = torch.sqrt(((u[:, i] + u[:, j]) ** 2).sum(-1).clamp_min(1e-30) / 4)
            s = torch.sqrt((1 - c * c + 1e-14).clamp_min(1e-30))
            d2 = torch.where(both, ((h[:, j] - h[:, i]) ** 2).sum(-1), torch.ones_like(c))
            Ri, Rj = R[ra[:, i]], R[ra[:, j]]
            e = ap[:, 2] * (1 - (ap[:, 0] * c + ap[:, 1] * s))
            e = e - _ljqh(d2, Ri[:, 0] + Rj[:, 0], Ri[:, 1] * Rj[:, 1], KE * Ri[:, 2] * Rj[:, 2],
                          (Ri[:, 3] * Rj[:, 3]).clamp_max(0))
            E = E + torch.where(both, e, torch.zeros_like(e))
    return E, sysn


def _pair_terms(b, pos, rcut):
    """Forces on atoms [nv, 3] and energies [nsys] of the pair term over the 9 images, molecules of like size together."""
    F = torch.zeros_like(pos)
    E = torch.zeros(b.nsys, device=_DEV, dtype=torch.float64)
    for ss, has, vi, ai in _chunks(b):
        N = has.shape[1]
        x, R = pos[torch.as_tensor(vi, device=_DEV)], _t(b.REQs[ai])
        live = torch.as_tensor(has, device=_DEV)
        ng = torch.as_tensor(np.where(has[..., None], b.neighs[ai], -1).astype(np.int64), device=_DEV)
        gc = torch.as_tensor(b.neighCell[ai].astype(np.int64), device=_DEV)
        R0 = R[:, :, None, 0] + R[:, None, :, 0]
        E0 = R[:, :, None, 1] * R[:, None, :, 1]
        Q = KE * R[:, :, None, 2] * R[:, None, :, 2]
        f = torch.zeros_like(x)
        e = torch.zeros(len(ss), device=_DEV, dtype=torch.float64)
        out0 = ~(live[:, :, None] & live[:, None, :]) | torch.eye(N, dtype=torch.bool, device=_DEV)
        for im in range(9):
            sh = torch.tensor([(im % 3 - 1) * CELL, (im // 3 - 1) * CELL, 0.0], device=_DEV, dtype=torch.float64)
            d = x[:, None, :, :] + sh - x[:, :, None, :]
            r2 = (d * d).sum(-1)
            out = out0.clone()
            for c in range(4):
                hit = (ng[:, :, c] >= 0) & (gc[:, :, c] == im)
                m = torch.zeros_like(out)
                m.scatter_(2, ng[:, :, c].clamp_min(0)[..., None], hit[..., None])
                out |= m
            if rcut > 0:
                out |= r2 >= rcut * rcut
            r2 = torch.where(out, torch.full_like(r2, 1e30), r2)
            ir2 = 1 / r2
            ir = torch.sqrt(ir2)
            u6 = (R0 * R0 * ir2) ** 3
            fr = -(12 * ir2 * (u6 - 1) * u6 * E0 + Q * ir * ir2)
            en = u6 * E0 * (u6 - 2) + Q * ir
            if rcut > 0:
                fr = fr + torch.where(out, torch.zeros_like(ir), Q * ir / rcut ** 2)
                en = en + torch.where(out, torch.zeros_like(ir), Q * (r2 * ir / rcut ** 2 - 2 / rcut))
            f += (d * fr[..., None]).sum(2)
            e += 0.5 * en.sum((1, 2))
        F[torch.as_tensor(vi[has], device=_DEV)] = f[live]
        E[torch.as_tensor(ss.copy(), device=_DEV)] = e
    return F, E


def _exact_eval(case, seed):
    k = _base(case)
    b = k["batch"]
    off = b.offsets()
    pos = _t(_geometry(k, seed, _noise(case))).requires_grad_(True)
    Eb, sysn = _bonded_energy(b, pos, off)
    F = -torch.autograd.grad(Eb.sum(), pos)[0]
    pos = pos.detach()
    atom = torch.as_tensor(k["atom"], device=_DEV)
    sysv = torch.as_tensor(k["sys"], device=_DEV)
    F = torch.where(atom[:, None], F, F - pos * (F * pos).sum(1, keepdim=True))
    Fp, Ep = _pair_terms(b, pos, case["rcut"])
    if "coefs" not in _kept:
        sub = _slab()
        _kept["coefs"] = (sub, _fit(_node_potentials(sub)))
    sub, C = _kept["coefs"]
    Fg, eg = _grid_terms(sub, C, pos[atom], _t(b.REQs))
    F += Fp
    F[atom] += Fg
    z = torch.zeros(b.nsys, device=_DEV, dtype=torch.float64)
    Ebs = z.clone().index_add_(0, torch.as_tensor(sysn, device=_DEV), Eb.detach())
    Egs = z.clone().index_add_(0, sysv[atom], eg)
    return dict(F=F.cpu().numpy(), E=torch.stack([Ebs, Ep, Egs, Ebs + Ep + Egs], 1).cpu().numpy())


def _exact_train(case, seed):
    F, T = _rows(case, seed)
    p = {n: _t(np.asarray(v, np.float32)) for n, v in _train_start().items()}
    istd = (np.float32(1) / np.maximum(_FSTD, np.float32(1e-6))).astype(np.float32)
    X = torch.zeros(case["rows"], 80, device=_DEV, dtype=torch.float64)
    X[:, :68] = (_t(F) - _t(_FMEAN)) * _t(istd)
    T = _t(T) / 0.2
    ntile = (case["rows"] + 127) // 128
    tiles = min(case["tiles"], ntile)
    m = {n: torch.zeros_like(v) for n, v in p.items()}
    s = {n: torch.zeros_like(v) for n, v in p.items()}
    keep = {n: torch.ones_like(v) for n, v in p.items()}
    keep["W1"][:, 68:] = 0
    keep["W3"][3:] = 0
    keep["b3"][3:] = 0
    losses, t0 = [], 0
    for t in range(1, case["steps"] + 1):
        if t0 + tiles > ntile:
            t0 = 0
        x, y = X[t0 * 128:(t0 + tiles) * 128], T[t0 * 128:(t0 + tiles) * 128]
        t0 += tiles
        n = x.shape[0]
        z1 = x @ p["W1"].T + p["b1"]
        s1 = torch.sigmoid(z1)
        z2 = (z1 * s1) @ p["W2"].T + p["b2"]
        s2 = torch.sigmoid(z2)
        d = (z2 * s2) @ p["W3"].T[:, :3] + p["b3"][:3] - y
        losses.append((d * d).sum() / n)
        dy = torch.zeros(n, 16, device=_DEV, dtype=torch.float64)
        dy[:, :3] = 2 * d / n
        g2 = (dy @ p["W3"]) * s2 * (1 + z2 * (1 - s2))
        g1 = (g2 @ p["W2"]) * s1 * (1 + z1 * (1 - s1))
        grad = {"W3": dy.T @ (z2 * s2), "b3": dy.sum(0), "W2": g2.T @ (z1 * s1), "b2": g2.sum(0), "W1": g1.T @ x,
                "b1": g1.sum(0)}
        for k in p:
            m[k] = 0.9 * m[k] + 0.1 * grad[k]
            s[k] = 0.999 * s[k] + 0.001 * grad[k] ** 2
            upd = (m[k] / (1 - 0.9 ** t)) / (torch.sqrt(s[k] / (1 - 0.999 ** t)) + 1e-8)
            if k[0] == "W":
                upd = upd + 0.01 * p[k]
            p[k] = (p[k] - 1e-3 * upd) * keep[k]
    return dict(losses=torch.stack(losses).cpu().numpy(), **{k: v.cpu().numpy() for k, v in p.items()})


def exact(case, seed):
    if case["kind"] == "eval":
        return _exact_eval(case, seed)
    if case["kind"] == "grid":
        return _fit(_node_potentials(prepare(case, seed)["sub"])).cpu().numpy()
    if case["kind"] == "train":
        return _exact_train(case, seed)
    # hundreds to thousands of steps over thousands of molecules: minutes in plain torch
    return None
