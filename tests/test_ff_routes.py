"""Which force-field calls are summed by boxes (ppgpu_ff_route, host only): that the GPU tests' cases
take the paths that they are there for, and what the rule does at its edges."""

import ctypes

import numpy as np
import pytest

from tests import test_gpu_ff_box as ffbox
from tests import test_gpu_tip_field as tipfield

LJ, COULOMB, LJC, QZS = 0, 1, 2, 3
WITH_E, ACCUMULATE, F64 = 1, 2, 4
TIP = dict(Qs=[-10.0, 20.0, -10.0, 0.0], QZs=[0.1, 0.0, -0.1, 0.0])


@pytest.fixture(scope="module")
def route():
    from ppafm_gb300 import _lib, build

    build.build()
    L = _lib.load()

    def fn(n, cell, natoms, ncharged, mode, kind=0, flags=0, ns=None):
        cell = np.diag(np.asarray(n) * cell) if np.isscalar(cell) else cell
        i = [np.ascontiguousarray(v, dtype=np.int32) for v in (n, n if ns is None else ns)]
        d = [np.ascontiguousarray(v, dtype=np.float64) for v in (cell, TIP["Qs"], TIP["QZs"])]
        out = np.full(2, -1, np.int32)
        ip, dp = (lambda a: a.ctypes.data_as(ctypes.POINTER(ctypes.c_int))), (lambda a: a.ctypes.data_as(ctypes.POINTER(ctypes.c_double)))
        _lib.check(L.ppgpu_ff_route(ip(i[0]), dp(d[0]), ip(i[1]), natoms, ncharged, mode, kind, dp(d[1]), dp(d[2]), flags, ip(out)))
        return tuple(int(v) for v in out)

    return fn


# (nodes, levels) of test_gpu_ff_box's CASES, in their order
FF_ROUTES = [
    (8, 0), (8, 0), (8, 0), (10, 1), (8, 0), (8, 0), (8, 0), (8, 0), (8, 0),
    (8, 1),
    (10, 1), (10, 1),  # near lists overflow; near atoms staged in parts
    (10, 3),  # levels and parents' lists
    (10, 2),  # 32-bit indices, no lists
    (8, 1), (8, 2),
    (8, 0),  # with the energy, 10 nodes take more atoms: MORE has them
    (10, 2), (10, 1), (8, 0), (8, 0), (10, 1),
]  # fmt: skip
MORE_ROUTES = [(10, 1)]


def _routes(route, cases):
    got = []
    for mode, n, step, tilt, natoms, kind, neutral, energy, acc in cases:
        rng = np.random.default_rng(natoms + n[0])
        cell = ffbox._cell(n, step, tilt)
        q = ffbox._atoms(rng, natoms, cell, kind)[2]
        q[rng.uniform(size=natoms) < neutral] = 0.0
        m = dict(ljc=LJC, lj=LJ, coulomb=COULOMB, qzs=QZS)[mode]
        nch = 0 if mode == "lj" else int((q != 0).sum())
        got.append(route(n, cell, natoms, nch, m, flags=WITH_E * energy + ACCUMULATE * acc))
    return got


def test_gpu_cases_take_their_paths(route):
    assert _routes(route, ffbox.CASES) == FF_ROUTES
    assert _routes(route, ffbox.MORE) == MORE_ROUTES


def test_gpu_tip_cases_take_their_paths(route):
    got = []
    for n, step, tilted, natoms, _, energy, acc in tipfield.BOXES:
        cell = np.diag(np.array(n) * step)
        if tilted:
            cell[1, 0], cell[2, 0], cell[2, 1] = 0.7, -0.9, 0.5
        got.append(route(n, cell, natoms, natoms, COULOMB, kind=2, flags=WITH_E * energy + ACCUMULATE * acc))
    assert got == [(10, 1), (10, 1), (10, 0), (10, 0), (10, 2), (10, 2), (10, 2), (10, 1)]
    for n2 in (1, 3, 33):  # the direct kernel's own cases
        assert route((9, 14, n2), tipfield.ORTHO, 513, 513, COULOMB, kind=1) == (0, 0)


def test_routes_of_small_and_float64_calls(route):
    assert route((40, 40, 40), 0.1, 342, 342, LJC) == (0, 0)  # 27 boxes
    assert route((200, 200, 200), 0.1, 342, 342, LJC, ns=(3, 3, 200)) == (0, 0)  # a sub-box of a grid by boxes
    assert route((200, 200, 200), 0.1, 342, 342, LJC) == (8, 1)
    assert route((200, 200, 200), 0.1, 342, 342, LJC, flags=F64) == (0, 0)
    assert route((200, 200, 200), 0.1, 0, 0, LJC) == (0, 0)
    assert route((200, 200, 200), 0.1, 342, 342, LJC, ns=(0, 200, 200)) == (0, 0)


@pytest.mark.parametrize("mode", [LJ, COULOMB, LJC, QZS])
@pytest.mark.parametrize("n", [(1, 2000, 2000), (2000, 1, 2000), (1, 1, 20000), (2, 1, 20000), (1500, 1, 400), (1, 300, 300)])
def test_planes_and_lines_go_pair_by_pair(route, mode, n):
    """Their leaves have fewer points than a box has nodes: by boxes they took 3 to 20 times as long."""
    for natoms in (60, 342, 1500, 18540):
        for flags in (0, WITH_E, ACCUMULATE):
            assert route(n, 0.1, natoms, natoms, mode, flags=flags) == (0, 0)
            assert route(n, 0.1, natoms, natoms, COULOMB, kind=2, flags=flags) == (0, 0)
    # a plane of a grid that itself goes by boxes
    assert route((200, 200, 200), 0.1, 342, 342, mode, ns=(1, 200, 200)) == (0, 0)


@pytest.mark.parametrize(
    "n,step,natoms,mode,want",
    [
        ((6, 400, 400), 0.1, 18540, LJ, (8, 2)),  # leaves of 1536 points
        ((4, 400, 400), 0.1, 1500, LJC, (8, 1)),  # 1024 points: no room for 6 x 250 cells of 10 nodes
        ((2, 400, 400), 0.1, 1500, LJC, (0, 0)),  # 512 points: nor of 8
        ((51, 32, 136), 0.335, 3869, LJC, (0, 0)),  # few boxes, most atoms within their reach
        ((101, 101, 63), 0.396, 18540, LJC, (10, 1)),  # few boxes, atoms far beyond it
        ((23, 188, 258), 0.468, 63, LJC, (0, 0)),  # 10 nodes for their shorter reach: few atoms
        ((192, 194, 178), 0.47, 297, LJC, (10, 1)),
    ],
)
def test_route_by_points_boxes_and_reach(route, n, step, natoms, mode, want):
    assert route(n, step, natoms, natoms if mode != LJ else 0, mode) == want
