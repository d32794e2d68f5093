"""The pz and dz2 tips' double-float kernel against the float64 twin (PPGPU_FF_F64) on the same
records, at the edges of its launch: columns shorter than, equal to and past a thread's 4
points, atom counts around the 256-atom tile, tilted cells, sub-boxes and accumulation.

Tolerance: both store float32 (2^-24 of the value each, 2^-23 together); a term's double-float
error is below 2^-42 of the Coulomb fields it subtracts, q/r^2 with weights summing to 20 (pz) or
400 (dz2).  Accumulating adds one more float32 rounding of the sum to each side (2^-23 in all)."""

import numpy as np
import pytest

from tests.conftest import grid_coords

pytestmark = pytest.mark.gpu

ORTHO = np.diag([4.2, 3.9, 5.1])
TILTED = np.array([[4.2, 0, 0.1], [0.5, 3.9, 0], [0.3, -0.4, 5.1]])


@pytest.mark.parametrize("kind", [1, 2])
@pytest.mark.parametrize("cell", [ORTHO, TILTED], ids=["ortho", "tilted"])
@pytest.mark.parametrize("n2,natoms", [(1, 1), (3, 255), (4, 256), (5, 257), (33, 513), (31, 40)])
def test_tip_field_matches_float64(gpulib, kind, cell, n2, natoms):
    from ppafm_gb300 import device as D

    rng = np.random.default_rng(1000 * kind + n2 + natoms)
    n = np.array([9, 14, n2], np.int32)
    R = np.column_stack([rng.uniform(-12, 16, natoms), rng.uniform(-12, 16, natoms), rng.uniform(-6, 0.4, natoms)])
    q = rng.uniform(-0.3, 0.3, natoms) * 14.399645
    atoms, na, nch = D.pack_atoms(R, None, q)
    ff = D.DeviceFF(n, cell)

    def run(f64, accumulate):
        ff.FE.fill_(0.25)
        return ff.compute(atoms, na, nch, D.FF_COULOMB, kind=kind, with_E=True, accumulate=accumulate, f64=f64).grid4.cpu().numpy().astype(np.float64)

    P = grid_coords(n, np.vstack([np.zeros(3), cell]))(np.indices(n).reshape(3, -1).T)[:, None]
    w = 20.0 if kind == 1 else 400.0
    r2 = np.maximum(((P - R[None]) ** 2).sum(-1), 1e-8)
    floor = (w * np.abs(q) / r2).sum(1) * 2.0**-42
    floor_E = (w * np.abs(q) / np.sqrt(r2)).sum(1) * 2.0**-42
    for accumulate in (False, True):
        got, ref = run(False, accumulate).reshape(-1, 4), run(True, accumulate).reshape(-1, 4)
        tol = 2.0**-23 * np.abs(ref) + np.column_stack([floor, floor, floor, floor_E])
        if accumulate:
            tol += 2.0**-23 * (np.abs(ref) + 0.25)
        assert (np.abs(got - ref) <= tol).all(), (accumulate, float((np.abs(got - ref) / tol).max()))
    i0, ns = (2, 3, 0), (5, 7, n2)
    whole = run(False, False)
    sub = ff.compute_subgrid(i0, ns, atoms, na, nch, D.FF_COULOMB, kind=kind, with_E=True).view(*ns, 4).cpu().numpy()
    assert (sub == whole[2:7, 3:10].astype(np.float32)).all()


BOXES = [
    # n, step, tilted, charges, spread in z, energy, accumulate
    ((113, 97, 130), 0.1, False, 200, 0.3, True, False),
    ((113, 97, 130), 0.1, True, 200, 0.3, False, False),
    ((97, 113, 128), 0.07, False, 300, 0.3, False, True),
    ((97, 113, 128), 0.07, True, 300, 0.3, True, True),
    ((180, 177, 161), 0.1, False, 400, 0.3, True, False),  # a level above the leaves
    ((180, 177, 161), 0.1, False, 400, 0.3, False, False),
    ((113, 112, 97), 0.1, False, 3000, 8.0, False, False),  # more near charges than the list holds
    ((113, 112, 97), 0.1, True, 900, 8.0, True, False),  # near charges staged in parts
]


@pytest.mark.parametrize("kind", [1, 2])
@pytest.mark.parametrize("case", BOXES, ids=lambda c: "-".join(map(str, c)))
def test_tip_boxes_match_float64(gpulib, kind, case):
    """The same tips by boxes, on sub-boxes of the grid: as above, and 1e-9 of the pairs' own fields
    (below 6 q / r^3 for pz, 20 q / r^4 for dz2) for the interpolation of the far ones."""
    import torch

    from ppafm_gb300 import device as D

    n, step, tilted, natoms, dz, energy, accumulate = case
    rng = np.random.default_rng(natoms + n[0])
    cell = np.diag(np.array(n) * step)
    if tilted:
        cell[1, 0], cell[2, 0], cell[2, 1] = 0.7, -0.9, 0.5
    L = np.diag(cell)
    R = np.column_stack([rng.uniform(-0.7 * L[0], 1.7 * L[0], natoms), rng.uniform(-0.7 * L[1], 1.7 * L[1], natoms), rng.uniform(-dz, 0.3, natoms)])
    if dz > 1:
        R[:, :2] = L[:2] / 2 + rng.normal(0, 2.5, (natoms, 2))
    q = rng.uniform(-0.3, 0.3, natoms) * 14.399645
    atoms, na, nch = D.pack_atoms(R, None, q)
    ff = D.DeviceFF(n, cell)
    ff.FE.fill_(0.25 if accumulate else float("nan"))
    got = ff.compute(atoms, na, nch, D.FF_COULOMB, kind=kind, with_E=energy, accumulate=accumulate).grid4.cpu().numpy().astype(np.float64)
    assert np.isfinite(got).all()
    ns = (5, 6, 9)
    corners = [(0, 0, 0)] + [tuple(int(rng.integers(0, n[k] - ns[k] + 1)) for k in range(3)) for _ in range(8)] + [tuple(n[k] - ns[k] for k in range(3))]
    w = 20.0 if kind == 1 else 400.0
    for i0 in corners:
        ref = ff.compute_subgrid(i0, ns, atoms, na, nch, D.FF_COULOMB, kind=kind, with_E=True, f64=True).view(-1, 4).cpu().numpy().astype(np.float64)
        g = got[i0[0] : i0[0] + 5, i0[1] : i0[1] + 6, i0[2] : i0[2] + 9].reshape(-1, 4)
        P = (np.indices(ns).reshape(3, -1).T + np.array(i0)) @ (cell / np.array(n)[:, None])
        r = np.sqrt(np.maximum(((P[:, None] - R[None]) ** 2).sum(-1), 1e-8))
        pair = 6 * np.abs(q) / r**3 if kind == 1 else 20 * np.abs(q) / r**4
        floor = (w * np.abs(q) / r**2).sum(1) * 2.0**-42 + 1e-9 * pair.sum(1)
        floor_E = (w * np.abs(q) / r).sum(1) * 2.0**-42 + 1e-9 * (pair * r).sum(1)
        tol = 2.0**-23 * np.abs(ref) + np.column_stack([floor, floor, floor, floor_E])
        if accumulate:
            tol += 2.0**-23 * (np.abs(ref) + 0.25)
            ref = ref + 0.25
        k = 4 if energy else 3
        d = np.abs(g - ref)
        assert (d[:, :k] <= tol[:, :k]).all(), (i0, float((d[:, :k] / tol[:, :k]).max()))
        if not energy:
            assert (g[:, 3] == (0.25 if accumulate else 0.0)).all()
    assert torch.isfinite(ff.FE).all()


@pytest.mark.parametrize("kind", [1, 2])
def test_tip_boxes_wide_indices(gpulib, kind):
    """More than 65536 charges, so that boxes list their near ones as 32-bit indices and hand no lists
    down; most of the charges below the grid, the others a plane in it.  Tolerance as above."""
    from ppafm_gb300 import device as D

    rng = np.random.default_rng(66000 + kind)
    n = np.array([113, 112, 97], np.int32)
    cell = np.diag(n * 0.1)
    R = np.column_stack([rng.uniform(-8, 19, (66000, 2)), rng.uniform(-60, -14, 66000)])
    R[-400:, 2] = rng.uniform(0.2, 0.8, 400)  # the highest indices are the near ones
    q = rng.uniform(-0.3, 0.3, len(R)) * 14.399645
    atoms, na, nch = D.pack_atoms(R, None, q)
    ff = D.DeviceFF(n, cell)
    ff.FE.fill_(float("nan"))
    got = ff.compute(atoms, na, nch, D.FF_COULOMB, kind=kind, with_E=True).grid4.cpu().numpy().astype(np.float64)
    assert np.isfinite(got).all()
    ns = (3, 4, 9)
    w = 20.0 if kind == 1 else 400.0
    for i0 in [(0, 0, 0), (50, 61, 3), (17, 90, 40), (110, 108, 88)]:
        ref = ff.compute_subgrid(i0, ns, atoms, na, nch, D.FF_COULOMB, kind=kind, with_E=True, f64=True).view(-1, 4).cpu().numpy().astype(np.float64)
        g = got[i0[0] : i0[0] + 3, i0[1] : i0[1] + 4, i0[2] : i0[2] + 9].reshape(-1, 4)
        P = (np.indices(ns).reshape(3, -1).T + np.array(i0)) * 0.1
        floor, floor_E = np.zeros(len(P)), np.zeros(len(P))
        for k, p in enumerate(P):
            r = np.sqrt(np.maximum(((p - R) ** 2).sum(1), 1e-8))
            pair = 6 * np.abs(q) / r**3 if kind == 1 else 20 * np.abs(q) / r**4
            floor[k] = (w * np.abs(q) / r**2).sum() * 2.0**-42 + 1e-9 * pair.sum()
            floor_E[k] = (w * np.abs(q) / r).sum() * 2.0**-42 + 1e-9 * (pair * r).sum()
        tol = 2.0**-23 * np.abs(ref) + np.column_stack([floor, floor, floor, floor_E])
        d = np.abs(g - ref)
        assert (d <= tol).all(), (i0, float((d / tol).max()))


@pytest.mark.parametrize("kind", [1, 2])
@pytest.mark.parametrize("n", [(9, 14, 33), (113, 97, 130)], ids=["pairs", "boxes"])
def test_a_charge_beyond_float32_adds_nothing(gpulib, kind, n):
    """A charge at 1e20 A, whose r^2 overflows float32: the bits of the field of the others, in place of
    the first charge's record a second one that is too far to show."""
    import torch

    from ppafm_gb300 import device as D

    rng = np.random.default_rng(77)
    cell = np.diag(np.array(n) * 0.1)
    R = np.column_stack([rng.uniform(-4, 15, 200), rng.uniform(-4, 15, 200), rng.uniform(-3, -0.5, 200)])
    q = rng.uniform(-0.3, 0.3, 200) * 14.399645
    got = []
    for far in (1e16, 1e20, -3e37):  # at 1e16 A q / r^3 is below float32's least as well
        R[11] = (far, 0.3 * far, 0.0)
        rec, na, nch = D.pack_atoms(R, None, q)
        got.append(D.DeviceFF(n, cell).compute(rec, na, nch, D.FF_COULOMB, kind=kind, with_E=True).FE.clone())
    assert torch.isfinite(got[0]).all() and got[1].equal(got[0]) and got[2].equal(got[0])
