"""Force fields by boxes (near atoms at the points, far ones on Chebyshev nodes) against the
float64 twin (PPGPU_FF_F64) on sub-boxes of the same grid: ragged sizes, tilted cells, every mode,
energies, accumulation, near lists that overflow their space, 32-bit atom indices, several levels,
atoms on grid points.

Tolerance: the force-field tests' own bar for float32 grids (tests.conftest.check_ff): within 1e-5
of max(|F|, 1e-2 eV/A), or, where the terms cancel, within 2^-20 of the sum of their magnitudes; the
interpolation of a far term is good to 1.5e-7 of it.  The tip-charge sums (AFMulator) subtract terms
two orders larger than the result: 5e-5, as in the direct kernel's test.  Energies: 1e-4, likewise.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

U = 2.0**-20


def _cell(n, step, tilt):
    c = np.diag(np.asarray(n) * step)
    if tilt:
        c[1, 0], c[2, 0], c[2, 1] = 0.1 * c[1, 1], 0.12 * c[2, 2], -0.07 * c[2, 2]
    return c


def _atoms(rng, natoms, cell, kind):
    L = np.diag(cell)
    if kind == "plane":  # a molecule and its images
        R = np.column_stack([rng.uniform(-L[0], 2 * L[0], natoms), rng.uniform(-L[1], 2 * L[1], natoms), rng.uniform(-0.3, 0.3, natoms)])
    elif kind == "slab":
        R = np.column_stack([rng.uniform(-L[0], 2 * L[0], natoms), rng.uniform(-L[1], 2 * L[1], natoms), rng.uniform(-15, 0.0, natoms)])
    else:  # "ball": most of them near every box
        R = np.asarray(cell).sum(0) / 2 + rng.normal(0, 2.5, (natoms, 3)) - np.array([0, 0, 0.5 * L[2] + 6.0])
    c = np.column_stack([rng.uniform(10, 60, natoms), rng.uniform(1e4, 8e4, natoms)])
    q = rng.uniform(-0.3, 0.3, natoms) * 14.399645
    return R, c, q


CASES = [
    # mode, n, step, tilt, atoms, kind, neutral share, energy, accumulate
    ("ljc", (113, 129, 97), 0.1, False, 130, "plane", 0.0, False, False),
    ("ljc", (113, 129, 97), 0.1, True, 130, "plane", 0.5, True, False),
    ("ljc", (128, 112, 130), 0.06, False, 400, "plane", 0.3, False, True),
    ("lj", (97, 161, 81), 0.14, False, 300, "plane", 1.0, True, False),
    ("lj", (97, 161, 81), 0.14, True, 300, "plane", 1.0, False, True),
    ("coulomb", (145, 113, 65), 0.1, False, 257, "plane", 0.0, True, False),
    ("coulomb", (145, 113, 65), 0.1, True, 200, "plane", 0.4, False, False),
    ("qzs", (130, 120, 110), 0.1, False, 40, "plane", 0.2, True, False),
    ("qzs", (130, 120, 110), 0.1, True, 40, "plane", 0.0, False, True),
    ("ljc", (200, 113, 129), 0.1, False, 700, "plane", 0.2, True, False),  # one level above the leaves
    ("lj", (113, 120, 113), 0.1, False, 3000, "ball", 1.0, False, False),  # near lists overflow
    ("ljc", (113, 120, 113), 0.1, False, 900, "ball", 0.1, False, False),  # near atoms staged in parts
    ("ljc", (250, 310, 330), 0.1, False, 20000, "slab", 0.97, False, False),  # two levels, parents' lists
    ("lj", (120, 113, 128), 0.1, False, 66000, "slab", 1.0, False, False),  # 32-bit indices, no lists
    ("ljc", (200, 157, 160), 0.1, True, 400, "plane", 0.3, True, False),  # 8 nodes, one level
    ("lj", (230, 225, 221), 0.1, False, 1000, "plane", 1.0, False, False),  # 8 nodes, two levels
    ("ljc", (113, 129, 97), 0.1, True, 300, "plane", 0.5, True, False),  # 10 nodes, one level
    ("ljc", (200, 200, 170), 0.1, False, 4500, "slab", 0.5, True, False),  # 10 nodes, two levels
    ("qzs", (130, 120, 110), 0.1, False, 300, "plane", 0.0, False, False),
    ("lj", (145, 113, 65), 0.1, True, 257, "plane", 1.0, True, False),
    ("coulomb", (145, 113, 65), 0.3, False, 257, "plane", 0.4, False, False),
    ("ljc", (113, 129, 97), 0.45, False, 130, "plane", 0.2, False, False),  # 10 nodes for their shorter reach
]


@pytest.mark.parametrize("case", CASES, ids=lambda c: "-".join(map(str, (c[0], *c[1], c[4], c[5], "tilt" if c[3] else "ortho", "E" if c[7] else "", "acc" if c[8] else ""))))
def test_boxes_match_float64(gpulib, case):
    from ppafm_gb300 import device as D

    mode, n, step, tilt, natoms, kind, neutral, energy, acc = case
    rng = np.random.default_rng(natoms + n[0])
    cell = _cell(n, step, tilt)
    R, c, q = _atoms(rng, natoms, cell, kind)
    q[rng.uniform(size=natoms) < neutral] = 0.0
    Q, Fmax = (-0.05, 10.0) if mode == "ljc" else (0.0, 0.0)
    tip = dict(Qs=[-10.0, 20.0, -10.0, 0.0], QZs=[0.1, 0.0, -0.1, 0.0]) if mode == "qzs" else {}
    M = dict(ljc=D.FF_LJC, lj=D.FF_LJ, coulomb=D.FF_COULOMB, qzs=D.FF_QZS)[mode]
    rec, na, nch = D.pack_atoms(R, None if mode == "coulomb" else c, None if mode == "lj" else q)
    ff = D.DeviceFF(n, cell)
    ff.FE.fill_(0.125 if acc else float("nan"))
    got = ff.compute(rec, na, nch, M, Q=Q, Fmax=Fmax, with_E=energy, accumulate=acc, **tip).grid4.cpu().numpy().astype(np.float64)
    assert np.isfinite(got).all()
    if acc:
        got -= 0.125
    sub = D.DeviceFF(n, cell, FE=ff.FE)
    corners = [(0, 0, 0)] + [tuple(int(rng.integers(0, n[k] - (6, 5, 9)[k] + 1)) for k in range(3)) for _ in range(8)] + [tuple(n[k] - (6, 5, 9)[k] for k in range(3))]
    for i0 in corners:
        ns = (6, 5, 9)
        flags = D.FF_F64 | (D.FF_WITH_E if energy else 0)
        ref = _subgrid_f64(sub, i0, ns, rec, na, nch, M, Q, Fmax, flags, tip)
        g = got[i0[0] : i0[0] + 6, i0[1] : i0[1] + 5, i0[2] : i0[2] + 9]
        P = (np.indices(ns).reshape(3, -1).T + np.array(i0)) @ (cell / np.array(n)[:, None])
        SF, SE = np.zeros(len(P)), np.zeros(len(P))
        for k, p in enumerate(P):
            r2 = ((p - R) ** 2).sum(1) + 1e-8
            i6 = r2**-3.0
            if mode != "coulomb":
                SF[k] += (np.abs(12 * c[:, 1] * i6) + np.abs(6 * c[:, 0])) @ (i6 * r2**-0.5)
                SE[k] += (c[:, 1] * i6 + c[:, 0]) @ i6
            if mode in ("ljc", "coulomb"):
                w = abs(Q) if mode == "ljc" else 1.0
                SF[k] += w * (np.abs(q) / r2).sum()
                SE[k] += w * (np.abs(q) * r2**-0.5).sum()
        F, G = ref[..., :3].reshape(-1, 3), g[..., :3].reshape(-1, 3)
        tol = np.maximum(U * SF, (5e-5 if mode == "qzs" else 1e-5) * np.maximum(np.linalg.norm(F, axis=1), 1e-2))
        ok = np.linalg.norm(F, axis=1) < 1e30
        d = np.linalg.norm(F - G, axis=1)
        assert (d[ok] <= tol[ok]).all(), (case, i0, float((d[ok] / tol[ok]).max()))
        if energy:
            tol = np.maximum(U * SE, 1e-4 * np.maximum(np.abs(ref[..., 3].ravel()), 1e-2))
            d = np.abs(ref[..., 3].ravel() - g[..., 3].ravel())
            assert (d[ok] <= tol[ok]).all(), (case, i0, "E", float((d[ok] / tol[ok]).max()))
        elif not acc:
            assert (g[..., 3] == 0).all()


MORE = [
    ("ljc", (113, 129, 97), 0.1, True, 1300, "plane", 0.5, True, False),  # 10 nodes with the energy, a tilted cell
]


@pytest.mark.parametrize("case", MORE, ids=lambda c: "-".join(map(str, (c[0], *c[1], c[4], c[5]))))
def test_more_boxes_match_float64(gpulib, case):
    test_boxes_match_float64(gpulib, case)


REPULSIVE = [
    ("lj", (130, 129, 113), 0.1, False, 200, "plane", 1.0, True, False),  # 8 nodes
    ("ljc", (113, 129, 97), 0.1, True, 260, "plane", 0.5, False, True),
    ("lj", (160, 113, 128), 0.1, False, 3000, "slab", 1.0, False, False),  # 10 nodes and levels
    ("ljc", (113, 129, 97), 0.1, False, 1300, "slab", 0.7, True, False),
]


@pytest.mark.parametrize("share", [0.5, 1.0])
@pytest.mark.parametrize("case", REPULSIVE, ids=lambda c: "-".join(map(str, (c[0], *c[1], c[4], c[5]))))
def test_atoms_without_attraction(gpulib, monkeypatch, case, share):
    """c6 = 0 for a share of the atoms: far from a distance at which the r^-13 force itself is
    interpolated to 1.5e-7.  Same tolerance."""
    import sys

    whole = _atoms

    def some(rng, natoms, cell, kind):
        R, c, q = whole(rng, natoms, cell, kind)
        c[: int(share * natoms), 0] = 0.0
        return R, c, q

    monkeypatch.setattr(sys.modules[__name__], "_atoms", some)
    test_boxes_match_float64(gpulib, case)


def test_atoms_without_attraction_are_far(gpulib):
    """They are left to the nodes like others: the field of 18540 of them takes a few times that of
    attractive ones (all near, it took 30 times as long and longer than pair by pair)."""
    import torch

    from ppafm_gb300 import device as D

    n, cell = (200, 200, 200), np.diag([20.0, 20.0, 20.0])
    R, c, _ = _atoms(np.random.default_rng(4), 18540, cell, "slab")
    ff = D.DeviceFF(n, cell)
    ms = []
    for c6 in (1.0, 0.0):
        rec, na, _ = D.pack_atoms(R, c * [c6, 1.0], None)
        t = []
        for _ in range(6):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            ff.compute(rec, na, 0, D.FF_LJ)
            b.record()
            b.synchronize()
            t.append(a.elapsed_time(b))
        ms.append(min(t))
    assert ms[1] < 8.0 * ms[0], ms


@pytest.mark.parametrize("mode", ["lj", "ljc", "coulomb"])
def test_an_atom_beyond_float32_adds_nothing(gpulib, mode):
    """An atom at 1e20 A, whose r^2 overflows: the bits of the field with that atom at 1e19 A, whose
    force is below float32's least."""
    from ppafm_gb300 import device as D

    n = (113, 129, 97)
    cell = np.diag(np.array(n) * 0.1)
    R, c, q = _atoms(np.random.default_rng(31), 300, cell, "plane")
    M = dict(ljc=D.FF_LJC, lj=D.FF_LJ, coulomb=D.FF_COULOMB)[mode]
    got = []
    for x in (1e19, 1e20):
        R[11] = (x, 0.0, 0.0)
        rec, na, nch = D.pack_atoms(R, None if mode == "coulomb" else c, None if mode == "lj" else q)
        got.append(D.DeviceFF(n, cell).compute(rec, na, nch, M, Q=-0.05 if mode == "ljc" else 0.0).FE.clone())
    assert bool(got[0].isfinite().all()) and got[1].equal(got[0])


def test_tip_charges_and_an_atom_beyond_float32(gpulib):
    """The same with a tip's charges, whose differences overflow there: every point goes through all atoms,
    as pair by pair (a small sub-box), bit for bit."""
    from ppafm_gb300 import device as D

    n = (113, 129, 97)
    cell = np.diag(np.array(n) * 0.1)
    R, c, q = _atoms(np.random.default_rng(33), 100, cell, "plane")
    R[11] = (1e20, 0.0, 0.0)
    tip = dict(Qs=[-10.0, 20.0, -10.0, 0.0], QZs=[0.1, 0.0, -0.1, 0.0])
    rec, na, nch = D.pack_atoms(R, c, q)
    ff = D.DeviceFF(n, cell)
    g = ff.compute(rec, na, nch, D.FF_QZS, with_E=True, **tip).grid4.cpu().numpy().astype(np.float64)
    assert np.isfinite(g).all()
    for i0 in [(0, 0, 0), (50, 60, 40), (107, 124, 88)]:
        ref = _subgrid_f64(ff, i0, (6, 5, 9), rec, na, nch, D.FF_QZS, 0.0, 0.0, D.FF_WITH_E, tip)
        assert (g[i0[0] : i0[0] + 6, i0[1] : i0[1] + 5, i0[2] : i0[2] + 9] == ref).all()


def test_infinite_charge_as_pair_by_pair(gpulib):
    """The same infinities and NaNs as the direct sum's (a small sub-box), bit for bit elsewhere too: all
    points take its slow path."""
    import torch

    from ppafm_gb300 import device as D

    n = (113, 129, 97)
    cell = np.diag(np.array(n) * 0.1)
    R, _, q = _atoms(np.random.default_rng(32), 300, cell, "plane")
    q[7] = np.inf
    R[7] = (300.0, 2.0, 5.0)
    rec, na, nch = D.pack_atoms(R, None, q)
    ff = D.DeviceFF(n, cell)
    g = ff.compute(rec, na, nch, D.FF_COULOMB, with_E=True).grid4
    for i0 in [(0, 0, 0), (50, 60, 40), (107, 124, 88)]:
        ref = ff.compute_subgrid(i0, (6, 5, 9), rec, na, nch, D.FF_COULOMB, with_E=True).view(6, 5, 9, 4)
        got = g[i0[0] : i0[0] + 6, i0[1] : i0[1] + 5, i0[2] : i0[2] + 9]
        assert torch.equal(got.isnan(), ref.isnan()) and torch.equal(got.nan_to_num(nan=0.0), ref.nan_to_num(nan=0.0))


def _subgrid_f64(ff, i0, ns, rec, na, nch, mode, Q, Fmax, flags, tip):
    """A sub-box of the grid in float64 (compute_subgrid has no tip charges)."""
    import torch

    from ppafm_gb300._lib import check, dptr, iptr, lib, stream_handle, tptr

    out = torch.empty(int(np.prod(ns)) * 4, dtype=torch.float32, device="cuda")
    qs, qz = (np.array(tip[k]) if tip else None for k in ("Qs", "QZs"))
    check(lib().ppgpu_ff_subgrid(tptr(out), iptr(ff.n), dptr(ff.cell), iptr(np.array(i0, np.int32)), iptr(np.array(ns, np.int32)), tptr(rec), na, nch, mode, 0, Q, Fmax, dptr(qs), dptr(qz), flags, stream_handle(None)))
    return out.view(*ns, 4).cpu().numpy().astype(np.float64)


def test_boxes_atoms_on_grid_points(gpulib):
    """Atoms on grid nodes, where float32 overflows: the clamped field of the direct kernel (a small
    sub-box of the same grid), node by node."""
    from ppafm_gb300 import device as D

    n, step = np.array([128, 128, 128]), 0.125
    cell = np.diag(n * step)
    rng = np.random.default_rng(3)
    R, c, q = _atoms(rng, 200, cell, "plane")
    nodes = rng.integers(2, 126, (20, 3))
    R[:20] = nodes * step
    rec, na, nch = D.pack_atoms(R, c, q)
    ff = D.DeviceFF(n, cell)
    g = ff.compute(rec, na, nch, D.FF_LJC, Q=-0.05, Fmax=10.0).grid4.cpu().numpy()
    assert np.isfinite(g).all()
    for x, y, z in nodes:
        ref = ff.compute_subgrid((x - 1, y - 1, z - 1), (3, 3, 3), rec, na, nch, D.FF_LJC, Q=-0.05, Fmax=10.0).view(3, 3, 3, 4).cpu().numpy()
        assert np.abs(g[x - 1 : x + 2, y - 1 : y + 2, z - 1 : z + 2] - ref).max() <= 1e-5 * 10.0


@pytest.mark.parametrize("tilt", [False, True])
def test_points_near_an_atom(gpulib, tilt):
    """Grid points 0.03 to 0.06 A from an atom, whose r^-14 shows the rounding of the displacement: its
    float32 rounding and the reciprocal root's (2^-22.9), 14 times, are 3e-6 of the force and energy."""
    from ppafm_gb300 import device as D

    n = (113, 129, 97)
    rng = np.random.default_rng(21)
    cell = _cell(n, 0.1, tilt)
    R, c, q = _atoms(rng, 300, cell, "plane")
    c = np.abs(c)
    nodes = np.column_stack([rng.integers(2, n[k] - 2, 24) for k in range(3)])
    d = rng.normal(size=(24, 3))
    R[:24] = nodes @ (cell / np.array(n)[:, None]) + d / np.linalg.norm(d, axis=1)[:, None] * rng.uniform(0.03, 0.06, (24, 1))
    rec, na, nch = D.pack_atoms(R, c, None)
    ff = D.DeviceFF(n, cell)
    g = ff.compute(rec, na, nch, D.FF_LJ, with_E=True).grid4.cpu().numpy().astype(np.float64)
    for x, y, z in nodes:
        ref = ff.compute_subgrid((int(x), int(y), int(z)), (1, 1, 1), rec, na, nch, D.FF_LJ, with_E=True, f64=True).view(4).cpu().numpy().astype(np.float64)
        got = g[x, y, z]
        assert np.linalg.norm(got[:3] - ref[:3]) <= 4e-6 * np.linalg.norm(ref[:3])
        assert abs(got[3] - ref[3]) <= 4e-6 * abs(ref[3])


def test_boxes_repeat_bit_for_bit(gpulib):
    from ppafm_gb300 import device as D

    n, cell = (160, 144, 150), np.diag([16.0, 14.4, 15.0])
    R, c, q = _atoms(np.random.default_rng(9), 600, cell, "plane")
    rec, na, nch = D.pack_atoms(R, c, q)
    ff = D.DeviceFF(n, cell)
    a = ff.compute(rec, na, nch, D.FF_LJC, Q=-0.05, Fmax=10.0).FE.clone()
    ff.FE.fill_(7.0)
    assert ff.compute(rec, na, nch, D.FF_LJC, Q=-0.05, Fmax=10.0).FE.equal(a)
