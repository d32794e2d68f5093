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
