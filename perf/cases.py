"""The work that a user of this library has it do, as cases that can be timed and compared.

A case is one call, or one short run of calls, through the public entry points, on inputs that
a user's program holds beforehand:

  scan       the whole pipeline of one system (force field, relaxed scan, df)
  field      a force-field grid of a molecule (LJ + Coulomb, LJ alone, Coulomb alone)
  slab       the same of a metal slab with a molecule on it: thousands of atoms, few charged
  tip_field  the Coulomb grid of a pz or dz2 tip
  relax      the relaxed scan over a given grid, with Fz -> df
  strokes    the reference's own entry point relaxTipStrokes_omp, host arrays in and out
  density    the density-overlap force field (FFT route)
  forces     potential2forces in float64, the default of the host entry point
  afm_field  the AFMulator's point-charge force field
  afm_scan   the AFMulator's relaxation and z convolution over a given grid
  hartree    the AFMulator's Hartree force field

Force fields and relaxations are separate cases, because a relaxation stops anywhere inside the
|F| < 1e-4 eV/A ball: the last bit of a force moves a stopping point by up to 1e-2 A.  A batch of
molecules is, system by system, the work of field and relax.

Sizes are those of ppafm_gb300/workloads.py and the AFMulator's defaults, the 800x800x500 slab
grid at half its resolution; ragged and smaller ones come with draw().
"""

import math
import random

import numpy as np
import torch

from ppafm_gb300 import HighLevel, core, workloads
from ppafm_gb300.AFMulator import AFMulator
from ppafm_gb300.device import DeviceFF, pack_atoms, relax_scan
from ppafm_gb300.field import HartreePotential
from ppafm_gb300.fieldFFT import FFTGrid
from ppafm_gb300.HighLevel import DensityOverlapPipeline, Pipeline, tip_vector
from ppafm_gb300._lib import FF_COULOMB, FF_LJ, FF_LJC

K_E = 14.399645  # eV A / e^2
EVA_NM = 16.0217662  # N/m per eV/A^2
FMAX = 10.0  # eV/A, the force clamp of the reference's stages
CHARGE = -0.05  # probe charge
# equilibrium radius (A) and well depth (eV) by element, and the oxygen probe's
SPECIES = {1: (1.487, 0.000681), 6: (1.908, 0.003729), 7: (1.78, 0.007372), 8: (1.6612, 0.009106), 9: (1.75, 0.002645), 17: (1.948, 0.011491), 79: (2.41, 0.01)}
PROBE_Z = 8
AFM_QS, AFM_QZS = (-10.0, 20.0, -10.0, 0.0), (0.1, 0.0, -0.1, 0.0)  # the AFMulator's default tip


def listed():
    return [
        # a quick look at a molecule: coarse grid, small scan; launches and the longest stroke count
        {"name": "scan_tiny", "kind": "scan", "n": 40, "npx": 32},
        # the field of the small-molecule workload: 38 charged atoms with their in-plane images
        {"name": "field_molecule", "kind": "field", "mode": "ljc", "n0": 200, "n1": 200, "n2": 200, "step": 0.1, "atoms": 38, "images": 1, "neutral": 0.0, "tilt": 0.0, "energy": False},
        # the largest: the slab workload (18 540 atoms with images) on 400x400x250 points
        {"name": "field_slab", "kind": "slab", "scale": 0.5},
        # a CO-like tip on the small molecule
        {"name": "field_dz2_tip", "kind": "tip_field", "tip": "dz2", "n0": 200, "n1": 200, "n2": 200, "step": 0.1, "atoms": 38, "images": 1},
        # the scan of the small-molecule workload
        {"name": "relax_molecule", "kind": "relax", "n": 200, "n2": 96, "step": 0.1, "atoms": 38, "npx": 160, "npy": 160, "nz": 30},
        # the scan of the slab workload: 262 144 strokes of 40 heights
        {"name": "relax_wide", "kind": "relax", "n": 400, "n2": 120, "step": 0.1, "atoms": 150, "npx": 512, "npy": 512, "nz": 40},
        # a program written for the reference's C core: host float64 grid and strokes
        {"name": "strokes_host", "kind": "strokes", "n": 96, "n2": 90, "step": 0.125, "atoms": 24, "npx": 64, "npy": 60, "nz": 20},
        # the density-overlap workload: 256^3 points, Pauli and Hartree parts
        {"name": "density_overlap", "kind": "density", "n": 256},
        # the host entry point's precision, on a ragged grid
        {"name": "forces_f64", "kind": "forces", "n0": 120, "n1": 108, "n2": 125},
        # one image of the training-set generator, its two halves; the AFMulator's default sizes
        {"name": "afm_field", "kind": "afm_field", "atoms": 38, "width": 16.0, "height": 3.0, "pix": 10},
        {"name": "afm_scan", "kind": "afm_scan", "atoms": 38, "width": 16.0, "npx": 128, "npy": 128, "nz": 30},
        # the same with electrostatics from a DFT Hartree potential
        {"name": "afm_hartree", "kind": "hartree", "atoms": 38, "width": 16.0, "pot": 150, "pix": 10},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng: random.Random):
    kind = rng.choice(["scan", "field", "field", "slab", "tip_field", "relax", "relax", "strokes", "density", "forces", "afm_field", "afm_scan", "hartree"])
    size = lambda lo, hi: int(round(_log(rng, lo, hi)))  # noqa: E731
    if kind == "scan":
        return {"kind": kind, "n": size(24, 64), "npx": size(8, 40)}
    if kind in ("field", "tip_field"):
        step = round(_log(rng, 0.05, 0.3), 4)
        c = {"kind": kind, "n0": size(32, 260), "n1": size(32, 260), "n2": size(24, 260), "step": step, "atoms": rng.randint(6, 60), "images": rng.choice([0, 1, 1])}
        if kind == "tip_field":
            return dict(c, tip=rng.choice(["pz", "dz2"]), n0=size(24, 160), n1=size(24, 160), n2=size(24, 160))
        return dict(c, mode=rng.choice(["ljc", "ljc", "lj", "coulomb"]), neutral=rng.choice([0.0, 0.0, 0.6]), tilt=rng.choice([0.0, 0.0, 0.15]), energy=rng.random() < 0.3)
    if kind == "slab":
        return {"kind": kind, "scale": round(_log(rng, 0.1, 0.45), 3)}
    if kind == "relax":
        return {"kind": kind, "n": size(100, 320), "n2": rng.randint(90, 120), "step": 0.1, "atoms": rng.randint(10, 60), "npx": size(16, 300), "npy": size(16, 300), "nz": rng.randint(12, 40)}
    if kind == "strokes":
        return {"kind": kind, "n": size(48, 120), "n2": rng.randint(70, 95), "step": 0.125, "atoms": rng.randint(10, 40), "npx": size(8, 80), "npy": size(8, 80), "nz": rng.randint(10, 30)}
    if kind == "density":
        return {"kind": kind, "n": size(64, 240)}
    if kind == "forces":
        return {"kind": kind, "n0": size(48, 140), "n1": size(48, 140), "n2": size(48, 140)}
    if kind == "afm_field":
        return {"kind": kind, "atoms": rng.randint(10, 60), "width": round(rng.uniform(6.0, 19.0), 1), "height": round(rng.uniform(1.5, 4.0), 1), "pix": rng.choice([8, 10, 10])}
    if kind == "afm_scan":
        return {"kind": kind, "atoms": rng.randint(10, 60), "width": 16.0, "npx": size(32, 160), "npy": size(32, 160), "nz": rng.randint(14, 34)}
    return {"kind": kind, "atoms": rng.randint(10, 60), "width": round(rng.uniform(8.0, 19.0), 1), "pot": size(80, 180), "pix": rng.choice([8, 10])}


# ------------------------------------------------------------------------------ inputs


def _molecule(rng, natoms, width, max_z=0.3):
    """natoms C/N/O/H/F/Cl atoms on a jittered honeycomb patch about the middle of a width x
    width square, z within max_z of 0: (Z [n], R [n, 3], Q [n] neutral)."""
    i, j = np.meshgrid(np.arange(-12, 13), np.arange(-12, 13), indexing="ij")
    a = 1.42 * math.sqrt(3.0)
    base = np.stack([i.ravel() * a + j.ravel() * a / 2, j.ravel() * a * math.sqrt(3.0) / 2], axis=1)
    sites = np.concatenate([base, base + np.array([0.0, 1.42])])
    near = np.argsort(np.linalg.norm(sites - rng.uniform(-1.0, 1.0, 2), axis=1), kind="stable")[:natoms]
    R = np.zeros((natoms, 3))
    R[:, :2] = sites[near] + rng.uniform(-0.1, 0.1, (natoms, 2)) + width / 2
    R[:, 2] = rng.uniform(-max_z, max_z, natoms)
    Z = rng.choice([6, 7, 8, 1, 9, 17], natoms, p=[0.4, 0.1, 0.1, 0.3, 0.05, 0.05])
    Q = rng.uniform(-0.3, 0.3, natoms)
    return Z, R, Q - Q.mean()


def _lj(Z):
    """(c6, c12) of each atom against the probe."""
    r = np.array([SPECIES[int(z)][0] for z in Z]) + SPECIES[PROBE_Z][0]
    e = np.sqrt(np.array([SPECIES[int(z)][1] for z in Z]) * SPECIES[PROBE_Z][1])
    return np.stack([2 * e * r**6, e * r**12], axis=1)


def _images(R, c, q, a, b, m):
    """The atoms and their in-plane images, m cells each way."""
    s = [i * np.asarray(a) + j * np.asarray(b) for i in range(-m, m + 1) for j in range(-m, m + 1)]
    return np.concatenate([R + t for t in s]), np.tile(c, (len(s), 1)), np.tile(q, len(s))


def _field_inputs(case, seed):
    """(n, lvec, R, cLJ, kqq) of a field or tip_field case."""
    rng = np.random.default_rng(seed)
    n = (case["n0"], case["n1"], case["n2"])
    L = [k * case["step"] for k in n]
    lvec = np.array([[0.0, 0.0, 0.0], [L[0], 0, 0], [0, L[1], 0], [0, 0, L[2]]])
    t = case.get("tilt", 0.0)
    lvec[2, 0], lvec[3, 0], lvec[3, 1] = t * L[1], t * L[2], -0.5 * t * L[2]
    Z, R, Q = _molecule(rng, case["atoms"], 0.0)
    R[:, :2] += 0.5 * (lvec[1] + lvec[2])[:2]
    Q = np.where(np.arange(len(Q)) < case.get("neutral", 0.0) * len(Q), 0.0, Q)
    return (n, lvec) + _images(R, _lj(Z), Q * K_E, lvec[1], lvec[2], case["images"])


def _slab_inputs(case, seed):
    w = workloads.slab_molecule(seed=seed, scale=case["scale"])
    R, c, q = _images(w["Rs"], _lj(w["Zs"]), w["Qs"] * K_E, w["lvec"][1], w["lvec"][2], 1)
    return w["gridN"], w["lvec"], R - w["lvec"][0], c, q


def _points(n, lvec, lo, hi):
    """Grid points lo..hi-1 (C order) relative to the origin, float64 [hi - lo, 3]."""
    p = torch.arange(lo, hi, device="cuda")
    ijk = torch.stack([p // (n[1] * n[2]), (p // n[2]) % n[1], p % n[2]], dim=1).double()
    return ijk @ torch.tensor(np.asarray(lvec)[-3:] / np.array(n)[:, None], device="cuda")


def _sums(n, lvec, R, c, q, eps=1e-8, tips=((1.0, 0.0),)):
    """Lennard-Jones and Coulomb (force, energy) sums [npts, 4] over the atoms in float64; tips:
    the probe's charges (weight, height)."""
    R, c, q = (torch.tensor(np.asarray(v, dtype=np.float64), device="cuda") for v in (R, c, q))
    npts = int(np.prod(n))
    lj, el = (torch.empty((npts, 4), dtype=torch.float64, device="cuda") for _ in range(2))
    step = max(1, 30_000_000 // max(1, len(R)))
    for lo in range(0, npts, step):
        P = _points(n, lvec, lo, min(npts, lo + step))
        d = [P[:, k, None] - R[None, :, k] for k in range(3)]
        xy = d[0] * d[0] + d[1] * d[1]
        i2 = 1.0 / (xy + d[2] * d[2] + eps)
        i6 = i2**3
        f = (12 * c[:, 1] * i6 - 6 * c[:, 0]) * (i6 * i2)
        for k in range(3):
            lj[lo : lo + step, k] = (f * d[k]).sum(1)
        lj[lo : lo + step, 3] = ((c[:, 1] * i6 - c[:, 0]) * i6).sum(1)
        e = torch.zeros((len(P), 4), dtype=torch.float64, device="cuda")
        for w, h in tips:
            z = d[2] + h
            i1 = (xy + z * z + eps).rsqrt()
            g = i1**3 * (q * w)
            for k, v in enumerate((d[0], d[1], z)):
                e[:, k] += (g * v).sum(1)
            e[:, 3] += (i1 * (q * w)).sum(1)
        el[lo : lo + step] = e
    return lj, el


def _clamp(F):
    r = F[:, :3].norm(dim=1, keepdim=True)
    F[:, :3] *= torch.where(r > FMAX, FMAX / r, torch.ones_like(r))
    return F


def _mixed(n, lvec, R, c, q):
    """clamp(F_LJ) + Q clamp(F_el), no energy: what a relaxation reads."""
    lj, el = _sums(n, lvec, R, c, q)
    F = _clamp(lj) + CHARGE * _clamp(el)
    F[:, 3] = 0.0
    return F


def _scan_setup(case, seed):
    """A molecule under a scan of its whole cell, as the relaxation gets it: the grid starts 1.5 A
    above the atoms, the heights are those of the workloads.  (n, lvec, FE [npts, 4] float64,
    xs, ys, zs, relaxation parameters)."""
    rng = np.random.default_rng(seed)
    n = (case["n"], case["n"], case["n2"])
    L = case["n"] * case["step"]
    lvec = np.array([[0.0, 0.0, 0.0], [L, 0, 0], [0, L, 0], [0, 0, n[2] * case["step"]]])
    Z, R, Q = _molecule(rng, case["atoms"], L)
    R[:, 2] -= 1.5
    FE = _mixed(n, lvec, R, _lj(Z), Q * K_E)
    xs, ys = np.arange(case["npx"]) * (L / case["npx"]), np.arange(case["npy"]) * (L / case["npy"])
    zs = (5.5 + 0.1 * np.arange(case["nz"]))[::-1].copy()
    return n, lvec, FE, xs, ys, zs, tip_vector(dict(workloads.PROBE, **workloads.FIRE))


def _df_weights(dz):
    """Giessibl weights of a 1 A oscillation, times f0 / k0 (for np.convolve)."""
    m = int(math.ceil(1.0 / dz))
    t = np.linspace(-1 + 2 * m * dz, -1, m + 1)
    f = np.sqrt(np.clip(1 - t * t, 0, None))
    f[0] = f[-1] = 0.0
    f2 = (np.arccos(np.clip(-t, -1, 1)) - t * f) / 2
    f2[0], f2[-1] = np.pi / 2, 0.0
    df, df2 = f[:-1] - f[1:], f2[:-1] - f2[1:]
    w = np.zeros(m + 1)
    w[1:] = t[:-1] * df + df2
    w[:-1] -= t[1:] * df + df2
    d = workloads.DF
    return w / (np.pi * dz) * 16.0217656 * d["f0Cantilever"] / d["kCantilever"]


def _afm(case):
    """An AFMulator with its default tip; the scan window is width x width x height."""
    h, w = case.get("height", 3.0), case["width"]
    dims = (case.get("npx", 128), case.get("npy", 128), case.get("nz", 30))
    return AFMulator(pixPerAngstrome=case.get("pix", 10), scan_dim=dims, scan_window=((2.0, 2.0, 7.0), (2.0 + w, 2.0 + w, 7.0 + h)), df_steps=min(10, dims[2]))


def _afm_molecule(case, seed):
    """Atoms under the scan window, coordinates and charges exact in float32."""
    Z, R, Q = _molecule(np.random.default_rng(seed), case["atoms"], case["width"] + 4.0)
    return Z, R.astype(np.float32).astype(np.float64), Q.astype(np.float32).astype(np.float64)


def _overlap_workload(case, seed):
    return workloads.density_overlap(seed=seed, scale=case["n"] / 256)


def _gaussians(n, lvec, atoms):
    """Sum of normalised Gaussians, minimum image, float64 [n0, n1, n2] (orthogonal cells)."""
    L = [lvec[k + 1][k] for k in range(3)]
    out = torch.zeros(tuple(n), dtype=torch.float64, device="cuda")
    for x, y, z, s, w in atoms:
        g = []
        for k, v in enumerate((x, y, z)):
            t = torch.arange(n[k], device="cuda", dtype=torch.float64) * (L[k] / n[k]) - v
            g.append(torch.exp(-((t - L[k] * torch.round(t / L[k])) ** 2) / (2 * s * s)) / (s * math.sqrt(2 * math.pi)))
        out += w * torch.einsum("i,j,k->ijk", *g)
    return out


# ------------------------------------------------------------------------------ cases


def prepare(case, seed):
    kind = case["kind"]
    if kind == "scan":
        w = workloads.small_molecule(seed=seed)
        L, z0, dz, npx = 20.0, 7.0, 0.1, case["npx"]
        w.update(gridN=(case["n"],) * 3, scanMin=(0.0, 0.0, z0), scanMax=(L - L / npx, L - L / npx, z0 + 29 * dz), scanStep=(L / npx, L / npx, dz))
        return {"kind": kind, "pl": Pipeline(w["Zs"], w["Rs"], w["Qs"], w["lvec"], w["gridN"], w, relax={k: w[k] for k in workloads.FIRE})}
    if kind in ("field", "slab", "tip_field"):
        n, lvec, R, c, q = _slab_inputs(case, seed) if kind == "slab" else _field_inputs(case, seed)
        mode = case.get("mode", "coulomb" if kind == "tip_field" else "ljc")
        rec, na, nch = pack_atoms(R, None if mode == "coulomb" else c, None if mode == "lj" else q)
        return {"kind": kind, "mode": mode, "energy": case.get("energy", False), "tip": HighLevel.TIP_KINDS[case.get("tip", "s")], "ff": DeviceFF(n, lvec), "atoms": (rec, na, nch)}
    if kind in ("relax", "strokes"):
        n, lvec, FE, xs, ys, zs, prm = _scan_setup(case, seed)
        if kind == "strokes":
            tips = np.stack(np.meshgrid(xs, ys, zs, indexing="ij"), axis=-1)
            return {"kind": kind, "n": n, "cell": lvec[1:], "F": FE[:, :3].contiguous().cpu().numpy().reshape(*n, 3), "tips": tips, "rs": np.zeros_like(tips), "fs": np.zeros_like(tips), "prm": prm}
        ff = DeviceFF(n, lvec, FE=FE.float().reshape(-1))
        dev = [torch.tensor(v, device="cuda") for v in (xs, ys, zs)]
        return {"kind": kind, "ff": ff, "scan": dev, "prm": prm, "W": _df_weights(zs[0] - zs[1]), "out": {}}
    if kind == "density":
        w = _overlap_workload(case, seed)
        return {"kind": kind, "pl": DensityOverlapPipeline.from_workload(w)}
    if kind == "forces":
        n = (case["n0"], case["n1"], case["n2"])
        g = torch.Generator(device="cuda").manual_seed(seed)
        lvec = _forces_cell(n)
        V = _gaussians(n, lvec, _forces_atoms(n, lvec, seed)) + 1e-3 * torch.randn(n, generator=g, device="cuda", dtype=torch.float64)
        rho = _gaussians(n, lvec, [(0.0, 0.0, 0.0, 0.7, 1.0), (0.0, 0.0, 1.1, 0.6, -0.4)])
        fft = FFTGrid(n, f64=True)
        return {"kind": kind, "fft": fft, "V": V.float(), "rho": rho.float(), "lvec": lvec, "FE": torch.empty(fft.N * 4, dtype=torch.float32, device="cuda")}
    afm = _afm(case)
    Z, R, Q = _afm_molecule(case, seed)
    if kind == "afm_field":
        return {"kind": kind, "afm": afm, "mol": (R, Z, Q)}
    if kind == "afm_scan":
        ff = afm.prepareFF(R, Z, Q)
        lj, el = _sums([int(v) for v in afm.nDim], afm.lvec, R - afm.lvec[0], _lj(Z), Q * K_E, eps=1e-6, tips=tuple(zip(AFM_QS, AFM_QZS)))
        ff.FE.copy_(torch.nan_to_num(lj + el).clamp(-1e6, 1e6).float().reshape(-1))
        return {"kind": kind, "afm": afm}
    n = (case["pot"], case["pot"] + 7, case["pot"] - 9)
    lvec = _pot_cell(case)
    pot = HartreePotential(_potential(case, seed).float(), lvec)
    afm.setRho({"dz2": -0.1}, sigma=0.71)
    assert pot.shape == n
    return {"kind": kind, "afm": afm, "mol": (R, Z, pot), "cell": lvec[1:]}


def _forces_cell(n):
    L = [0.12 * v for v in n]
    return np.array([[0.0, 0, 0], [L[0], 0, 0], [0, L[1], 0], [0, 0, L[2]]])


def _forces_atoms(n, lvec, seed):
    rng = np.random.default_rng(seed)
    return [(*(rng.uniform(0, lvec[k + 1][k]) for k in range(3)), rng.uniform(0.4, 0.9), rng.uniform(-4, 4)) for _ in range(20)]


def _pot_cell(case):
    """The cell of a Hartree potential: the molecule's, wider than the scan window."""
    w = case["width"] + 8.0
    return np.array([[-2.0, -2.0, -6.0], [w, 0, 0], [0, w + 1.0, 0], [0, 0, 24.0]])


def _potential(case, seed):
    """A smooth periodic potential (V) of screened charges on the molecule's atoms."""
    n = (case["pot"], case["pot"] + 7, case["pot"] - 9)
    lvec = _pot_cell(case)
    _, R, Q = _afm_molecule(case, seed)
    return _gaussians(n, lvec, [(*(r - lvec[0]), 1.1, 12.0 * q) for r, q in zip(R, Q)])


def run(state):
    kind = state["kind"]
    if kind == "scan":
        return state["pl"].run()
    if kind in ("field", "slab", "tip_field"):
        ff, (rec, na, nch) = state["ff"], state["atoms"]
        if state["mode"] == "ljc":
            ff.compute(rec, na, nch, FF_LJC, Q=CHARGE, Fmax=FMAX, with_E=state["energy"])
        elif state["mode"] == "lj":
            ff.compute(rec, na, 0, FF_LJ, with_E=state["energy"]).clamp(FMAX)
        else:
            ff.compute(rec, na, nch, FF_COULOMB, kind=state["tip"], with_E=state["energy"]).clamp(FMAX)
        # without with_E the energy slot holds nothing that the entry point promises
        return ff.grid4 if state["energy"] else ff.grid4[..., :3]
    if kind == "relax":
        return relax_scan(state["ff"], state["prm"], *state["scan"], df_weights=state["W"], out=state["out"])
    if kind == "strokes":
        p = state["prm"]
        core.setGridN(state["n"])
        core.setGridCell(state["cell"])
        core.setFF_Fpointer(state["F"])
        core.setRelax(int(p[0]), p[1], p[2], p[3])
        core.setTip(p[7], p[8], p[9:12].copy(), p[12:15].copy())
        core.relaxTipStrokes_omp(state["tips"], state["rs"], state["fs"])
        return {"rs": state["rs"], "fs": state["fs"]}
    if kind == "density":
        return state["pl"].build_ff().grid4
    if kind == "forces":
        return state["fft"].potential2forces(state["V"], state["rho"], state["lvec"], FE=state["FE"])
    if kind == "afm_field":
        return state["afm"].prepareFF(*state["mol"]).grid4
    if kind == "afm_scan":
        return state["afm"].evalAFM(keep_device=True)
    return state["afm"].prepareFF(*state["mol"], sample_lvec=state["cell"]).grid4


def work(case):
    """Bytes: every input read once and every output written once.  Flops: 26 for each pair of a
    point and a neutral atom, 30 for a charged one, 20 more for each further tip charge; 250 for
    the one force evaluation that a height of a stroke cannot do without; 2.5 N log2 N for each
    real transform of the FFT routes."""
    kind = case["kind"]
    if kind == "scan":
        heights, na = case["npx"] ** 2 * 30, 342
        return {"bytes": 16.0 * case["n"] ** 3 + 24.0 * heights + 48 * na, "flops": 30.0 * na * case["n"] ** 3 + 250.0 * heights}
    if kind in ("field", "tip_field"):
        pts, na = case["n0"] * case["n1"] * case["n2"], case["atoms"] * (2 * case["images"] + 1) ** 2
        per = {"lj": 26.0, "coulomb": 14.0, "ljc": 30.0}[case.get("mode", "coulomb")] + (40.0 if case.get("tip") == "dz2" else 20.0 if kind == "tip_field" else 0.0)
        return {"bytes": 16.0 * pts + 48 * na, "flops": per * pts * na}
    if kind == "slab":
        pts = round(800 * case["scale"]) ** 2 * round(500 * case["scale"])
        return {"bytes": 16.0 * pts + 48 * 18540, "flops": pts * (26.0 * 18000 + 30.0 * 540)}
    if kind in ("relax", "strokes"):
        rows = min(case["n2"], int(0.1 * case["nz"] / case["step"]) + 8)  # heights of the grid that the probe visits
        grid, heights = case["n"] ** 2 * rows, case["npx"] * case["npy"] * case["nz"]
        return {"bytes": (16.0 * grid + 24.0 * heights) if kind == "relax" else (24.0 * grid + 72.0 * heights), "flops": 250.0 * heights}
    if kind == "density":
        N = float(case["n"] ** 3)
        return {"bytes": N * (3 * 4 + 16), "flops": 7 * 2.5 * N * math.log2(N)}
    if kind == "forces":
        N = float(case["n0"] * case["n1"] * case["n2"])
        return {"bytes": N * (2 * 4 + 16), "flops": 6 * 2.5 * N * math.log2(N)}
    if kind == "afm_scan":
        heights = case["npx"] * case["npy"] * case["nz"]
        return {"bytes": 16.0 * (10 * case["width"] + 60) ** 2 * 40 + 20.0 * heights, "flops": 250.0 * heights}
    sizes = [v for v in (16, 32, 64, 128, 192, 256, 384, 512)]
    up = lambda v: next(s for s in sizes if s >= round(v))  # noqa: E731
    side, tall = up(case["pix"] * (case["width"] + 6.0)), up(case["pix"] * (case.get("height", 3.0) + 10.0))
    pts = float(side * side * tall)
    if kind == "afm_field":
        return {"bytes": 16.0 * pts, "flops": (26.0 + 60.0) * pts * case["atoms"]}
    return {"bytes": 16.0 * pts + 4.0 * case["pot"] ** 3, "flops": 26.0 * pts * case["atoms"] * 9 + 2 * 2.5 * pts * math.log2(pts)}


# ------------------------------------------------------------------------------ in 64 bits


def _trilinear(FE, n, g):
    """Periodic trilinear interpolation of FE [n0, n1, n2, k] at grid coordinates g [p, 3]."""
    f = torch.floor(g)
    t, i = g - f, f.long()
    out = 0.0
    for b in range(8):
        k = [(b >> 2) & 1, (b >> 1) & 1, b & 1]
        w = math.prod((t[:, a] if k[a] else 1 - t[:, a]) for a in range(3))
        out = out + w[:, None] * FE[(i[:, 0] + k[0]) % n[0], (i[:, 1] + k[1]) % n[1], (i[:, 2] + k[2]) % n[2]]
    return out


def _fire_scan(FE, n, cell, xs, ys, zs, prm):
    """The reference core's strokes, all pixels at once: (r, F) [npix, nz, 3] in approach order."""
    iters, conv, dtmax, a0, finc, fdec, falpha, l0, kr = (float(v) for v in prm[:9])
    dev = FE.device
    r0, ks = torch.tensor(prm[9:12], device=dev), torch.tensor(prm[12:15], device=dev)
    M = torch.tensor(np.linalg.inv(np.asarray(cell)) * np.array(n)[None, :], device=dev)
    X, Y = np.meshgrid(xs, ys, indexing="ij")
    tip = torch.tensor(np.stack([X.ravel(), Y.ravel(), 0 * X.ravel()], axis=1), device=dev)
    d = r0.repeat(len(tip), 1)
    rs, fs = [], []
    for z in zs:
        tip[:, 2] = float(z)
        live = torch.arange(len(tip), device=dev)
        x, v = d.clone(), torch.zeros_like(d)
        dt, a = (torch.full((len(tip), 1), s, dtype=torch.float64, device=dev) for s in (dtmax, a0))
        for _ in range(int(iters)):
            p = x[live]
            l = p.norm(dim=1, keepdim=True)
            f = _trilinear(FE, n, (tip[live] + p) @ M) + p * (kr * (l - l0) / l) + (p - r0) * ks
            u, h, m = v[live], dt[live], a[live]
            ff, vv, vf = (f * f).sum(1, True), (u * u).sum(1, True), (f * u).sum(1, True)
            back = vf < 0
            mixed = u * (1 - m) + f * (m * torch.sqrt(vv / ff.clamp_min(1e-300)))
            u = torch.where(back, torch.zeros_like(u), mixed)
            h = torch.where(back, h * fdec, (h * finc).clamp_max(dtmax))
            m = torch.where(back, torch.full_like(m, a0), m * falpha)
            u = u + f * h
            x[live], v[live], dt[live], a[live] = p + u * h, u, h, m
            live = live[(ff[:, 0] >= conv)]
            if not len(live):
                break
        d = x
        rs.append(tip + d)
        fs.append(_trilinear(FE, n, (tip + d) @ M))
    return torch.stack(rs, 1), torch.stack(fs, 1)


def _scan_outputs(FE, n, lvec, xs, ys, zs, prm, W):
    r, F = _fire_scan(FE.double().reshape(*n, -1)[..., :3], n, np.asarray(lvec)[1:], xs, ys, zs, prm)
    shape = (len(xs), len(ys), len(zs))
    fz = F[:, :, 2].flip(1).reshape(shape)
    w = torch.tensor(W[::-1].copy(), device=fz.device)
    df = (fz.unfold(2, len(W), 1) * w).sum(-1)
    return {"fzs": fz, "ppos": r.flip(1).reshape(*shape, 3) + torch.tensor(np.asarray(lvec)[0], device=r.device), "df": df}


def _afm_image(FE, n, afm):
    """relaxStrokesTilted and the z convolution."""
    dev = FE.device
    dtmax, a0 = 0.5, 0.1
    ks = torch.tensor([0.25, 0.25, 0.0], dtype=torch.float64, device=dev) / -EVA_NM
    kr, l0, r0 = 30.0 / -EVA_NM, 3.0, torch.tensor([0.0, 0.0, -3.0], dtype=torch.float64, device=dev)
    M = torch.tensor(np.linalg.inv(afm.lvec[1:]) * np.array(n)[None, :], device=dev)
    (x0, y0, z0), (x1, y1, z1) = afm.scan_window
    nx, ny, nz = afm.scan_dim
    X, Y = np.meshgrid(np.linspace(x0, x1, nx), np.linspace(y0, y1, ny), indexing="ij")
    tip = np.stack([X.ravel(), Y.ravel(), np.full(X.size, z1)], axis=1) - afm.lvec[0]
    tip = torch.tensor(tip.astype(np.float32).astype(np.float64), device=dev)
    pos = tip + r0
    dt, a = (torch.full((len(tip), 1), s, dtype=torch.float64, device=dev) for s in (dtmax, a0))
    fz = []
    for _ in range(nz):
        v, live, got = torch.zeros_like(pos), torch.arange(len(tip), device=dev), torch.zeros(len(tip), dtype=torch.float64, device=dev)
        for _ in range(128):
            p, u, h, m = pos[live], v[live], dt[live], a[live]
            F = _trilinear(FE, n, p @ M)
            q = p - tip[live]
            r = q.norm(dim=1, keepdim=True)
            f = F + (q - r0) * ks + q * (kr * (r - l0) / r)
            ff, vv, vf = (f * f).sum(1, True), (u * u).sum(1, True), (f * u).sum(1, True)
            back = vf < 0
            u = torch.where(back, torch.zeros_like(u), u * (1 - m) + f * (m * torch.sqrt(vv / (ff + 1e-8))))
            h = torch.where(back, (h * 0.5).clamp_min(0.1 * dtmax), (h * 1.1).clamp_max(dtmax))
            m = torch.where(back, torch.full_like(m, a0), m * 0.99)
            u = u + f * h
            pos[live], v[live], dt[live], a[live], got[live] = p + u * h, u, h, m, F[:, 2]
            live = live[ff[:, 0] >= 1e-8]
            if not len(live):
                break
        fz.append(got)
        tip[:, 2] -= afm.dz
        pos[:, 2] -= afm.dz
    k = afm.df_steps
    t = np.linspace(-1 + 0.5 / k, 1 - 0.5 / k, k - 1)
    w = np.zeros(k)
    w[:-1] = np.sqrt(1 - t * t)
    w[1:] -= np.sqrt(1 - t * t)
    w = w / (np.sum(np.linspace(-1, 1, k) * w) * k * afm.dz) * EVA_NM * afm.f0Cantilever / afm.kCantilever
    F = torch.stack(fz, 1)
    return (F.unfold(1, k, 1) * torch.tensor(w, device=dev)).sum(-1).reshape(nx, ny, nz - k + 1)


def _rolled(n, L):
    """Coordinates of the rolled grid, the origin at index 0."""
    return [torch.tensor([(i if i < n[k] // 2 else i - n[k]) * L[k] / n[k] for i in range(n[k])], dtype=torch.float64, device="cuda") for k in range(3)]


def _overlap_forces(V, rho, lvec):
    """(Fx, Fy, Fz, E) of the cross-correlation of V with rho, complex FFTs (orthogonal cells)."""
    n = V.shape
    L = [lvec[k + 1][k] for k in range(3)]
    C = torch.fft.fftn(V) * torch.fft.fftn(rho).conj() * math.prod(L[k] / n[k] for k in range(3))
    out = []
    for k in range(3):
        # spatial frequency along axis k on the rolled index
        z = (_rolled(n, [float(v) for v in n])[k] / L[k]).reshape([-1 if a == k else 1 for a in range(3)])
        out.append(torch.fft.ifftn(C * z * (-2j * math.pi)).real)
    out.append(torch.fft.ifftn(C).real)
    return torch.stack(out, -1)


def _poisson(rho, lvec):
    n = rho.shape
    g2 = 0.0
    for k in range(3):
        m = torch.fft.fftfreq(n[k], 1.0 / n[k], device="cuda", dtype=torch.float64) * (2 * math.pi / lvec[k + 1][k])
        g2 = g2 + (m**2).reshape([-1 if a == k else 1 for a in range(3)])
    g2[0, 0, 0] = math.inf
    return torch.fft.ifftn(torch.fft.fftn(rho) * (4 * math.pi * K_E) / g2).real


def exact(case, seed):
    kind = case["kind"]
    if kind == "scan":
        s = prepare(case, seed)["pl"]  # the scan's coordinates and the atoms' images
        w = workloads.small_molecule(seed=seed)
        R, c, q = _images(w["Rs"], _lj(w["Zs"]), w["Qs"] * K_E, w["lvec"][1], w["lvec"][2], 1)
        FE = _mixed((case["n"],) * 3, w["lvec"], R, c, q)
        return _scan_outputs(FE, (case["n"],) * 3, w["lvec"], s.xs, s.ys, s.zs, tip_vector(w), _df_weights(0.1))
    if kind in ("field", "slab", "tip_field"):
        n, lvec, R, c, q = _slab_inputs(case, seed) if kind == "slab" else _field_inputs(case, seed)
        if len(R) * float(np.prod(n)) > 1.5e11:
            return None
        tips = {"pz": ((-10.0, -0.1), (10.0, 0.1)), "dz2": ((-200.0, 0.0), (100.0, -0.1), (100.0, 0.1))}.get(case.get("tip"), ((1.0, 0.0),))
        lj, el = _sums(n, lvec, R, c, q, tips=tips)
        mode = case.get("mode", "coulomb" if kind == "tip_field" else "ljc")
        F = _clamp(lj) + CHARGE * _clamp(el) if mode == "ljc" else _clamp(lj if mode == "lj" else el)
        F = F.reshape(*n, 4)
        return F if case.get("energy") else F[..., :3]
    if kind in ("relax", "strokes"):
        n, lvec, FE, xs, ys, zs, prm = _scan_setup(case, seed)
        if case["npx"] * case["npy"] * case["nz"] > 4_000_000:
            return None
        if kind == "strokes":
            r, F = _fire_scan(FE.reshape(*n, 4)[..., :3], n, lvec[1:], xs, ys, zs, prm)
            shape = (len(xs), len(ys), len(zs), 3)
            return {"rs": r.reshape(shape), "fs": F.reshape(shape)}
        return _scan_outputs(FE.float(), n, lvec, xs, ys, zs, prm, _df_weights(zs[0] - zs[1]))
    if kind == "density":
        w = _overlap_workload(case, seed)
        n, lvec = w["gridN"], w["lvec"]
        rel = lambda a: _gaussians(n, lvec, a)  # noqa: E731
        rho_s, rho_t = rel(w["rho_e_atoms"]), rel(w["tip_atoms"])
        rho_q = rel(w["core_atoms"]) - rho_s
        return w["Apauli"] * _overlap_forces(rho_s, rho_t, lvec) + w["charge"] / w["tip_electrons"] * _overlap_forces(_poisson(rho_q, lvec), rho_t, lvec)
    if kind == "forces":
        s = prepare(case, seed)
        return _overlap_forces(s["V"].double(), s["rho"].double(), s["lvec"]).reshape(-1)
    afm = _afm(case)
    n = [int(v) for v in afm.nDim]
    Z, R, Q = _afm_molecule(case, seed)
    lj, el = _sums(n, afm.lvec, R - afm.lvec[0], _lj(Z), Q * K_E, eps=1e-6, tips=tuple(zip(AFM_QS, AFM_QZS)))
    if kind == "afm_field":
        return (lj + el).reshape(*n, 4)
    if kind == "afm_scan":
        FE = torch.nan_to_num(lj + el).clamp(-1e6, 1e6).float().double()
        return _afm_image(FE.reshape(*n, 4)[..., :3], n, afm)
    lvec = _pot_cell(case)
    V = _potential(case, seed).float().double()
    m = tuple(V.shape)
    h = [afm.lvec[k + 1][k] / n[k] for k in range(3)]
    P = torch.stack(torch.meshgrid(*[(torch.arange(n[k], device="cuda").double() * h[k] + afm.lvec[0][k] - lvec[0][k]) * (m[k] / lvec[k + 1][k]) for k in range(3)], indexing="ij"), -1)
    E = torch.cat([_trilinear(V[..., None], m, g.reshape(-1, 3)) for g in P]).reshape(n)
    x, y, z = (v.reshape([-1 if a == k else 1 for a in range(3)]) / 0.71 for k, v in enumerate(_rolled(n, [afm.lvec[k + 1][k] for k in range(3)])))
    g = torch.exp(-(x * x + y * y + z * z) / 2)
    rho = -0.1 * 0.25 * (2 * z * z - x * x - y * y) * g / (g.sum() * math.prod(h))
    E = torch.fft.ifftn(torch.fft.fftn(E) * torch.fft.fftn(rho).conj()).real * math.prod(h)
    G = [(torch.roll(E, 1, k) - torch.roll(E, -1, k)) / (2 * h[k]) for k in range(3)]
    Ri, ci, qi = _images(R, _lj(Z), Q, lvec[1], lvec[2], 1)
    lj, _ = _sums(n, afm.lvec, Ri.astype(np.float32).astype(np.float64) - afm.lvec[0], ci, qi, eps=1e-6)
    return torch.stack(G + [E], -1) + lj.reshape(*n, 4)
