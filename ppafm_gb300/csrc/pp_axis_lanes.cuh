// pp_axis_lanes.cuh -- how relax_axis_kernel (pp_relax.cu) puts strokes on the lanes of a warp, and
// the grid offsets that its lanes exchange.  Plain C++ as well, so that the CPU tests run the same
// arithmetic over all 32 lanes.
#pragma once

#ifdef __CUDACC__
#define PP_AXIS_FN __host__ __device__ __forceinline__
#else
#define PP_AXIS_FN inline
#endif

namespace ppgpu {

constexpr int AXIS_STROKES = 10;  // per warp, three lanes each

// Two lanes of a warp are left over.  They run the loop as well and gather, for nothing, from the
// offsets that they are passed, so they read along with the last stroke's lanes: offsets of the
// three axes, as every address needs.
struct AxisLane {
    int grp, k;  // stroke of the warp, axis
    int l0;      // lane of the stroke's axis 0
    bool spare;  // left over: never active
};
PP_AXIS_FN AxisLane axis_lane(int lane) {
    AxisLane a;
    a.spare = lane >= 3 * AXIS_STROKES;
    a.grp = a.spare ? AXIS_STROKES - 1 : lane / 3;
    a.l0 = 3 * a.grp;
    a.k = lane % 3;
    return a;
}

// The lane that a value of axis a is read from.
PP_AXIS_FN int axis_source(const AxisLane &l, int a) { return l.l0 + a; }

// Points of the grid from its first one to corner j (bits: x, y, z) of a cell, from the offsets
// o[axis][0 or 1] of the cell's two planes along each axis; below the number of points when each
// axis's offset is its own.
PP_AXIS_FN int axis_corner(const int o[3][2], int j) { return o[0][j >> 2] + o[1][(j >> 1) & 1] + o[2][j & 1]; }

}  // namespace ppgpu
