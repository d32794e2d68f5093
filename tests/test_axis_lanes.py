"""The gathers of relax_axis_kernel (three lanes a stroke, two lanes of a warp left over) stay inside
the grid: the lane map and address arithmetic of csrc/pp_axis_lanes.cuh, compiled for the CPU and
run over all 32 lanes of a warp the way the kernel does (shuffle sources modulo the warp), with the
strokes' cells anywhere, ended and missing strokes, and the left-over lanes where a probe's rest
position without a tip puts them."""

import os
import shutil
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ppafm_gb300", "csrc")

HARNESS = r"""
#include "pp_axis_lanes.cuh"
using namespace ppgpu;
// n: grid; cells[32]: the cell of each lane along its own axis k.  Returns the number of gathers outside
// [0, n0 n1 n2), and of lanes whose offsets are not those of axes 0, 1, 2 of one stroke.
extern "C" int bad_gathers(const int *n, const int *cells, int *axis, int *group) {
    int a0[32], a1[32];
    for (int lane = 0; lane < 32; lane++) {
        const AxisLane l = axis_lane(lane);
        const int m = n[l.k], pitch = l.k == 0 ? n[1] * n[2] : (l.k == 1 ? n[2] : 1);
        const int i0 = cells[lane] % m, i1 = i0 + 1 == m ? 0 : i0 + 1;
        a0[lane] = i0 * pitch;
        a1[lane] = i1 * pitch;
        axis[lane] = l.k;
        group[lane] = l.spare ? -1 : l.grp;
    }
    const long long N = (long long)n[0] * n[1] * n[2];
    int bad = 0;
    for (int lane = 0; lane < 32; lane++) {
        const AxisLane l = axis_lane(lane);
        int o[3][2];
        for (int a = 0; a < 3; a++) {
            const int from = axis_source(l, a) % 32;
            bad += axis_lane(from).k != a;
            o[a][0] = a0[from];
            o[a][1] = a1[from];
        }
        for (int j = 0; j < 8; j++) {
            const long long at = axis_corner(o, j);
            bad += at < 0 || at >= N;
        }
    }
    return bad;
}
"""


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    import ctypes

    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    d = tmp_path_factory.mktemp("axis")
    src, so = d / "h.cpp", d / "h.so"
    src.write_text(HARNESS)
    subprocess.run([cxx, "-std=c++17", "-O1", "-shared", "-fPIC", "-I", CSRC, str(src), "-o", str(so)], check=True)
    fn = ctypes.CDLL(str(so)).bad_gathers
    p = np.ctypeslib.ndpointer(np.int32, flags="C")
    fn.argtypes = [p, p, p, p]
    return fn


@pytest.mark.parametrize("n", [(200, 200, 96), (128, 128, 128), (34, 29, 41), (1, 1, 1), (2, 3, 1), (1290, 1290, 1290)])
def test_gathers_stay_in_the_grid(harness, n):
    n = np.array(n, np.int32)
    axis, group = np.zeros(32, np.int32), np.zeros(32, np.int32)
    rng = np.random.default_rng(int(n.sum()))
    # rest positions (0, 0) and (+-0.1, +-0.1): cells 0 or n - 1 of the lanes that hold no stroke
    for spare in ([0, 0], [-1, 0], [0, -1], [-1, -1]):
        for first in range(0, int(n[0]), max(1, int(n[0]) // 40)):
            cells = rng.integers(0, 1 << 20, 32).astype(np.int32)
            cells[0] = first  # lane 0: x of the warp's first stroke, in every part of the grid
            cells[30:] = [int(n[k]) + s if s else 0 for k, s in enumerate(spare)]
            assert harness(n, cells, axis, group) == 0
        cells = np.array([n[lane % 3] - 1 for lane in range(32)], np.int32)  # the last cell of every axis
        assert harness(n, cells, axis, group) == 0
    # every stroke of a warp has its three axes once, and two lanes have none
    assert sorted((g, k) for g, k in zip(group, axis) if g >= 0) == [(g, k) for g in range(10) for k in range(3)]
    assert (group < 0).sum() == 2
