// pp_ff_box.cu -- force-field grids by boxes: near atoms point by point, far atoms on
// Chebyshev nodes.
//
// The field of an atom that is far from a box of grid points is smooth over the box, so it is
// summed on a few nodes and interpolated from there, instead of being summed at every point
// (the one-level form of the kernel-independent, interpolation-based fast summation: W. Fong and
// E. Darve, "The black-box fast multipole method", J. Comput. Phys. 228 (2009)).  The sums are
// those of ff_block (pp_ff_dev.cuh): the same pair interactions, in the same arithmetic.
//
//  * A leaf box is up to 16 x 16 x 16 points, one CTA.  Its far atoms are summed on 8 x 8 x 8
//    Chebyshev nodes (512 against 4096 points), its near ones at the points.
//  * Levels above it: boxes of 2 x 2 x 2 boxes of the level below, with the same 8^3 nodes, so
//    that atoms farther away cost 1/8 at each level.  An atom is summed at the highest level at
//    which it is far from the leaf's ancestor.  An upper box interpolates its nodes' sums to the
//    nodes of its 8 children, which start from them.
//  * Far at a level: R^2 >= (7 H)^2 from the box's centre, H its half diagonal.  The
//    interpolation error of the r^-7 force (dispersion, the steepest that matters at that
//    distance) is then below 1e-7 of the pair's force, under the ~4e-7 rounding of a float32
//    pair term.  The r^-13 repulsion needs more distance the stronger it is beside the
//    dispersion: an atom whose coefficients do not satisfy the bound in `far` stays near, whatever
//    they are.
//  * The interpolated sums handed to a child lie in the child's own part of the output grid until
//    its CTA reads them and later writes its points there: no workspace.  A box that is too small
//    to hold them (a remainder at the grid's edge), and every box when FE is accumulated into,
//    sums its far atoms itself.
//
// Bound by float32 FMA like ff_block, on far fewer pairs.  Figures beside ff_box_rule below.
#include <algorithm>
#include <cmath>
#include <cstring>

#include "pp_ff_box_dev.cuh"

namespace ppgpu {

constexpr int BOX_FOLD = 64;     // near atoms summed before they join a point's running sum
constexpr int BOX_P2 = 4;        // pairs of a thread's run of 8 nodes or points along z

// --------------------------------------------------------------------------- sums

template <int MODE, bool WITH_E>
struct BoxSums {
    static constexpr int U = (MODE == M_LJC) ? BOX_P2 : 1;
    static constexpr int NC1 = WITH_E ? 4 : 3;                   // components of one sum
    static constexpr int NC = (MODE == M_LJC) ? 2 * NC1 : NC1;   // LJC: LJ, then electrostatic
    Acc<BOX_P2> a;
    Acc<U> u;
    __device__ __forceinline__ void zero() {
        a.zero();
        u.zero();
    }
    // Component k (a constant after unrolling) of pair p.
    __device__ __forceinline__ float2 &at(int k, int p) {
        if (MODE == M_LJC && k >= NC1) {
            const int c = k - NC1, q = p < U ? p : 0;
            return c == 0 ? u.x[q] : (c == 1 ? u.y[q] : (c == 2 ? u.z[q] : u.e[q]));
        }
        return k == 0 ? a.x[p] : (k == 1 ? a.y[p] : (k == 2 ? a.z[p] : a.e[p]));
    }
};

// Adds one atom to the sums of a thread's 8 positions: the double-float position o and offsets
// from it, as floats (nodes: off[axis][i] in shared memory) or in two parts (POINT: B.offh, offl).
// Points can be close to the atom, where the rounding of their offsets would count.
template <int MODE, bool WITH_E, bool ORTHO, bool POINT>
__device__ __forceinline__ void box_add(const FFParams &prm, const BoxPrm &B, const dfl o[3], const float (*off)[8],
                                        const float4 &r0, const float4 &r1, const float4 &r2r, bool charged,
                                        BoxSums<MODE, WITH_E> &S) {
    const float eps = prm.eps;
    const float h[3] = {o[0].h + r0.x, o[1].h + r0.y, o[2].h + r1.x}, l[3] = {o[0].l + r0.z, o[1].l + r0.w, o[2].l + r1.y};
    const float2 c6n6 = bc(r1.z), c12x12 = bc(r1.w), c6n = bc(r2r.x), c12 = bc(r2r.y), kqq = bc(r2r.z);
    const float x0 = h[0] + l[0], y0 = h[1] + l[1], z0 = h[2] + l[2];
    const float2 xy0 = bc(fmaf(x0, x0, fmaf(y0, y0, eps)));
    auto along = [&](int k, float v0, int p) -> float2 {  // component k of pair p's displacement
        if constexpr (POINT)
            return add2(add2(bc(h[k]), make_float2(B.offh[k][2 * p], B.offh[k][2 * p + 1])),
                        add2(bc(l[k]), make_float2(B.offl[k][2 * p], B.offl[k][2 * p + 1])));
        else
            return add2(bc(v0), make_float2(off[k][2 * p], off[k][2 * p + 1]));
    };
#pragma unroll
    for (int p = 0; p < BOX_P2; p++) {
        const float2 dz = along(2, z0, p);
        const float2 dx = ORTHO ? bc(x0) : along(0, x0, p), dy = ORTHO ? bc(y0) : along(1, y0, p);
        const float2 xy = ORTHO ? xy0 : fma2(dy, dy, fma2(dx, dx, bc(eps)));
        const float2 r2 = fma2(dz, dz, xy);
        if constexpr (MODE == M_COUL) {
            const float2 ir = rsqrt2(r2);
            coul_ir<WITH_E, BOX_P2>(ir, mul2(ir, ir), dx, dy, dz, kqq, S.a, p);
        } else if constexpr (MODE == M_LJC) {
            if (charged)
                ljc_ir<WITH_E, BOX_P2>(rsqrt2(r2), dx, dy, dz, c6n6, c12x12, c6n, c12, kqq, S.a, S.u, p);
            else
                lj_ir2<WITH_E, BOX_P2>(rcp2(r2), dx, dy, dz, c6n6, c12x12, c6n, c12, S.a, p);
        } else {
            lj_ir2<WITH_E, BOX_P2>(rcp2(r2), dx, dy, dz, c6n6, c12x12, c6n, c12, S.a, p);
            if (MODE == M_QZS && charged) qzs_tip<WITH_E, BOX_P2>(prm, r2r.z, r2, dx, dy, dz, xy, S.a, p);
        }
    }
}

// Rare: a point whose float32 sums overflow, within ~5e-3 A of an atom: the far sums t (and u) and
// the near atoms (records in shared memory) with r^2 floored like ff_block's slow path.
template <int MODE, bool WITH_E>
__device__ __noinline__ float4 box_point_slow(const FFParams &prm, dfl x, dfl y, dfl z, const float4 *near, int nnear,
                                              int ncharged, float4 t, float4 u) {
    for (int j = 0; j < nnear; j++) {
        const float4 r0 = near[3 * j], r1 = near[3 * j + 1], r2r = near[3 * j + 2];
        const float dx = (x.h + r0.x) + (x.l + r0.z), dy = (y.h + r0.y) + (y.l + r0.w), dz = (z.h + r1.x) + (z.l + r1.y);
        const float dxy2 = fmaf(dx, dx, fmaf(dy, dy, prm.eps));
        const float r2 = fmaxf(fmaf(dz, dz, dxy2), R2CAP);
        const bool charged = j < ncharged;
        if (MODE != M_COUL) {
            const float ir2 = 1.f / r2, ir6 = ir2 * ir2 * ir2;
            const float fr = fmaf(r1.w, ir6, r1.z) * (ir6 * ir2);
            t.x = fmaf(fr, dx, t.x);
            t.y = fmaf(fr, dy, t.y);
            t.z = fmaf(fr, dz, t.z);
            t.w = fmaf(fmaf(r2r.y, ir6, r2r.x), ir6, t.w);
        }
        if (!charged) continue;
        const int nq = MODE == M_QZS ? prm.nqa : (MODE == M_LJ ? 0 : 1);
        for (int k = 0; k < nq; k++) {
            const float dq = MODE == M_QZS ? dz + prm.QZa[k] : dz;
            const float ir = rsqrtf(fmaxf(fmaf(dq, dq, dxy2), R2CAP));
            const float eq = r2r.z * ir * (MODE == M_QZS ? prm.Qa[k] : 1.f), fq = eq * ir * ir;
            float4 &a = MODE == M_LJC ? u : t;
            a.x = fmaf(fq, dx, a.x);
            a.y = fmaf(fq, dy, a.y);
            a.z = fmaf(fq, dq, a.z);
            a.w += eq;
        }
    }
    return finalize<MODE, WITH_E>(t.x, t.y, t.z, t.w, u.x, u.y, u.z, u.w, prm);
}

// ------------------------------------------------------------------------- the kernel

// Two tiles of NT atoms or the nodes' sums, and the running sums or the lines along x.
template <int MODE, bool WITH_E, int NT>
__host__ __device__ constexpr size_t box_tiles() {
    constexpr size_t t = sizeof(float4) * 2 * NT * FF_REC, n = sizeof(float) * BoxSums<MODE, WITH_E>::NC * BOX_N3;
    return t > n ? t : n;
}
// ... and, behind the lines, a leaf's running sums of the points (LJ, or the only sum).
template <int MODE, bool WITH_E, int NT>
constexpr size_t box_smem() {
    using S = BoxSums<MODE, WITH_E>;
    constexpr size_t sums = sizeof(float2) * S::NC * BOX_P2 * NT, lines = sizeof(float) * S::NC * BOX_S * 64 + sizeof(float2) * S::NC1 * BOX_P2 * NT;
    return box_tiles<MODE, WITH_E, NT>() + (NT == BOX_NT && lines > sums ? lines : sums);
}

// Leaves in CTAs of 256 threads: the warps of a scheduler then run the same part of the long
// straight-line code (with 128, four CTAs at four places waited on instruction fetches), two CTAs
// a SM at 128 registers.  Upper boxes with 128 or 256 (launch_box).
template <int MODE, bool WITH_E, bool ORTHO, bool LEAF, int NT>
__global__ void __launch_bounds__(NT, 512 / NT) ff_box_kernel(const __grid_constant__ FFParams prm, const __grid_constant__ BoxPrm B) {
    static_assert(!LEAF || NT == BOX_NT, "the leaves' tables are laid out for 256 threads");
    constexpr int SUBS = NT / 64;
    using Sums = BoxSums<MODE, WITH_E>;
    constexpr int NC = Sums::NC;
    // tiles: two atom tiles, then the nodes' sums, then the near atoms.  part: each thread's
    // running sums over the tiles, then the nodes' sums interpolated along x.
    extern __shared__ __align__(128) unsigned char box_raw[];
    float4 *tiles = reinterpret_cast<float4 *>(box_raw);
    float2 *part = reinterpret_cast<float2 *>(box_raw + box_tiles<MODE, WITH_E, NT>());
    __shared__ uint64_t bar[2];
    __shared__ unsigned short s_near[LEAF ? BOX_NEAR : 1];
    __shared__ unsigned short s_left[NT];  // upper boxes: a tile's atoms for the children
    __shared__ BoxPick<NT> pk;
    __shared__ dfl s_node[3][BOX_N][3];          // node positions: the parts along each axis (z: the middle only)
    __shared__ dfl s_pt[3][BOX_S][3];            // the points', runs along z from their middle (LEAF)
    __shared__ float s_off[3][8];                // offsets of the nodes along z
    __shared__ __align__(16) float s_wx[BOX_S][BOX_N], s_wy[BOX_S][BOX_N], s_wz[2][BOX_N][8];

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int level = LEAF ? 0 : B.level;
    const int nat = (MODE == M_COUL) ? prm.ncharged : prm.natoms;
    const int ntiles = (nat + NT - 1) / NT;
    int b[3], lo[3], hi[3];
    box_of_cta(prm, B, level, b, lo, hi);
    BoxShare share;
    bool handed = false;  // the parent's sums are there
    int nlist = -1;       // atoms that the parent left to this box (-1: no list)
    if (level < B.levels) {
        share = box_share<NC>(prm, B, level, b);
        handed = share_has_slot<NC>(share, level);
        if (handed && share.room > 0) nlist = *share_count(share, level);
    }
    const int nanc = handed ? B.levels - level : 0;
    const int ncand = nlist >= 0 ? nlist : nat, ncand_tiles = (ncand + NT - 1) / NT;
    auto fetch = [&](int t) {
        const int nj = min(NT, nat - t * NT);
        const uint32_t bytes = (uint32_t)nj * FF_REC * 16u;
        mbar_expect_tx(&bar[t & 1], bytes);
        bulk_g2s(tiles + (t & 1) * NT * FF_REC, prm.atoms + (size_t)t * NT * FF_REC, bytes, &bar[t & 1]);
    };
    if (tid == 0) {
        mbar_init(&bar[0], 1);
        mbar_init(&bar[1], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        if (nlist < 0)
            for (int t = 0; t < 2 && t < ntiles; t++) fetch(t);
    }
    // ---- tables of this box
    if (warp == 1 && lane <= nanc) pk.centre[lane] = box_centre(prm, B, level, b, lane);
    if (warp == 0 && lane < 24) {  // (middle + half t_i) steps
        const int a = lane >> 3, i = lane & 7;
        int l, h;
        box_span(prm, B, level, a, a == 0 ? b[0] : (a == 1 ? b[1] : b[2]), l, h);
        const float mid = 0.5f * (float)(l + h) + (float)prm.i0[a];
        const dfl e = df_mul_f(cheb_t(i), box_half(l, h)), g = a < 2 ? df_add(e, {mid, 0.f}) : dfl{mid, 0.f};
#pragma unroll
        for (int k = 0; k < 3; k++) {
            s_node[a][i][k] = df_mul(B.step[a][k], g);
            if (a == 2) s_off[k][i] = df_round(df_mul(B.step[2][k], e));
        }
    }
    if constexpr (LEAF) {
        if (warp >= 2 && warp < 4 && tid - 64 < 34) {
            const int i = tid - 64, a = i >> 4, j = i & 15;
            const float g = (float)(prm.i0[a] + (a == 0 ? lo[0] : (a == 1 ? lo[1] : lo[2])) + j) + (a == 2 ? 7.f : 0.f);
#pragma unroll
            for (int k = 0; k < 3; k++) s_pt[a][j][k] = df_mul_f(B.step[a][k], g);
        }
        if (tid >= 128) {
            const int pt = (tid - 128) / BOX_N, k = tid % BOX_N;
            s_wx[pt][k] = c_cheb_points.w[hi[0] - lo[0] + 1][pt][k];
            s_wy[pt][k] = c_cheb_points.w[hi[1] - lo[1] + 1][pt][k];
            s_wz[pt & 1][k][pt >> 1] = c_cheb_points.w[hi[2] - lo[2] + 1][pt][k];
        }
    } else {  // the children's nodes in this box: child c of an axis, its node pt & 7
        for (int i = tid; i < 3 * BOX_S * BOX_N; i += NT) {
            const int a = i / (BOX_S * BOX_N), pt = (i / BOX_N) % BOX_S, k = i % BOX_N;
            const float w = df_round(box_child_weight(prm, B, level, a, a == 0 ? b[0] : (a == 1 ? b[1] : b[2]), pt, k));
            if (a == 0) s_wx[pt][k] = w;
            if (a == 1) s_wy[pt][k] = w;
            if (a == 2) s_wz[pt >> 3][k][pt & 7] = w;
        }
    }
    // ---- far atoms on the nodes: thread = node column (ia, ib), one of SUBS parts of the atoms
    const int sub = tid >> 6, col = tid & 63;
    Sums S;
    S.zero();
#pragma unroll
    for (int k = 0; k < NC; k++)
#pragma unroll
        for (int p = 0; p < BOX_P2; p++) part[(k * BOX_P2 + p) * NT + tid] = make_float2(0.f, 0.f);
    __syncthreads();
    dfl on[3];
#pragma unroll
    for (int k = 0; k < 3; k++) on[k] = df_add(df_add(s_node[0][col >> 3][k], s_node[1][col & 7][k]), s_node[2][0][k]);
    const bool wide = nat > 65536;  // near indices as int
    const int near_cap = wide ? BOX_NEAR / 2 : BOX_NEAR;
    auto near_at = [&](int i) -> int { return wide ? reinterpret_cast<const int *>(s_near)[i] : (int)s_near[i]; };
    int nmid = 0, nzero = 0, place = -1;
    auto pick = [&](const float4 *T, int nj, int want, bool ok) {
        return box_pick<MODE, NT>(B, pk, level, nanc, T, nj, want, ok, nmid, nzero, place);
    };
    // This thread's atom of tile t of the parent's list, or (all) of all atoms, into the tile.  The
    // list is gone once the box writes its points.
    auto gather = [&](int t, bool all) -> int {
        const int i = t * NT + tid;
        int j = -1;
        if (i < (all ? nat : ncand)) {
            j = all ? i : (int)*share_list(share, level, i);
            box_gather(prm, tiles + ((t & 1) * NT + tid) * FF_REC, j);
        }
        return j;
    };
    int nnear = 0, nch = 0;  // atoms of class 0, charged ones among them
    for (int t = 0; t < ncand_tiles; t++) {
        const int base = t * NT;
        const float4 *T = tiles + (t & 1) * NT * FF_REC;
        int j0 = base + tid;
        bool landed = true;
        if (nlist >= 0)
            j0 = gather(t, false);  // each thread classifies what it gathered
        else
            landed = mbar_wait_bounded(&bar[t & 1], (uint32_t)(t >> 1) & 1u);
        if (!pick(T, min(NT, ncand - base), 1, landed)) {
            if (tid == 0) {
                raise_device_error(prm.err, PPGPU_ERR_DEVICE_TIMEOUT);
                for (int u = t; u < t + 2 && u < ntiles; u++) mbar_wait_bounded(&bar[u & 1], (uint32_t)(u >> 1) & 1u);
            }
            return;
        }
        if (place >= 0) {
            if constexpr (LEAF) {
                const int i = nnear + place;
                if (i < near_cap) {
                    if (wide) reinterpret_cast<int *>(s_near)[i] = j0;
                    else s_near[i] = (unsigned short)j0;
                }
            } else {
                s_left[place] = (unsigned short)j0;
            }
        }
        __syncthreads();
        if constexpr (!LEAF) box_leave<NC, NT>(prm, B, level, b, s_left, nzero, nnear);
        nnear += nzero;
        for (int i = sub; i < nmid; i += SUBS) {
            const int j = pk.mid[i];
            const float4 r2r = T[3 * j + 2];
            const bool charged = nlist >= 0 ? r2r.w != 0.f : base + j < prm.ncharged;
            box_add<MODE, WITH_E, ORTHO, false>(prm, B, on, s_off, T[3 * j], T[3 * j + 1], r2r, charged, S);
        }
        if (nmid > 0) {  // running sums over the tiles (two-level summation)
#pragma unroll
            for (int k = 0; k < NC; k++)
#pragma unroll
                for (int p = 0; p < BOX_P2; p++) {
                    float2 &r = part[(k * BOX_P2 + p) * NT + tid];
                    r = add2(r, S.at(k, p));
                }
            S.zero();
        }
        __syncthreads();
        if (nlist < 0 && tid == 0 && t + 2 < ntiles) fetch(t + 2);
    }
    if constexpr (!LEAF) box_leave_count<NC>(prm, B, level, b, nnear);
    __syncthreads();
    // ---- the nodes' sums: of all parts of the atoms and the parent's interpolated sums
    float4 *nodes = tiles;  // [NC][8][8][8]
    for (int k = sub; k < NC; k += SUBS) {
        float2 r[BOX_P2];
#pragma unroll
        for (int p = 0; p < BOX_P2; p++) {
            const float2 *v = part + (k * BOX_P2 + p) * NT + col;
            r[p] = add2(v[0], v[64]);
            if constexpr (SUBS == 4) r[p] = add2(r[p], add2(v[128], v[192]));
        }
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int e = k * (BOX_N3 / 4) + 2 * col + h;
            float4 v = make_float4(r[2 * h].x, r[2 * h].y, r[2 * h + 1].x, r[2 * h + 1].y);
            if (handed) {
                const float4 o = *share_slot<NC>(share, level, e);
                v = make_float4(v.x + o.x, v.y + o.y, v.z + o.z, v.w + o.w);
            }
            nodes[e] = v;
        }
    }
    __syncthreads();
    // ---- interpolated along x: line[k][x][ib][ic]
    float4 *line = reinterpret_cast<float4 *>(part);
    for (int i = tid; i < NC * 32; i += NT) {
        const int k = i >> 5, r = i & 15, x0 = (i & 16) ? BOX_S / 2 : 0;  // r: (ib, half of ic)
        float4 v[BOX_N];
#pragma unroll
        for (int a = 0; a < BOX_N; a++) v[a] = nodes[k * (BOX_N3 / 4) + a * 16 + r];
#pragma unroll 2
        for (int x = x0; x < x0 + BOX_S / 2; x++) {
            float2 s0 = make_float2(0.f, 0.f), s1 = s0;
#pragma unroll
            for (int a = 0; a < BOX_N; a++) {
                const float2 w = bc(s_wx[x][a]);
                s0 = fma2(w, make_float2(v[a].x, v[a].y), s0);
                s1 = fma2(w, make_float2(v[a].z, v[a].w), s1);
            }
            line[(k * BOX_S + x) * 16 + r] = make_float4(s0.x, s0.y, s1.x, s1.y);
        }
    }
    __syncthreads();
    // Near atoms first..last-1 of the list into the tiles' space (the nodes' sums are done with).
    auto stage = [&](int first, int last) {
        for (int i = tid; i < (last - first) * FF_REC; i += NT)
            tiles[i] = ldg4(prm.atoms + (size_t)near_at(first + i / FF_REC) * FF_REC + i % FF_REC);
        __syncthreads();
    };
    const bool listed = nnear <= near_cap, staged = nnear <= BOX_STAGE;
    if (LEAF && listed) {
        for (int i0 = 0; i0 < nnear; i0 += NT) {  // the charged ones come first
            const int i = i0 + tid;
            nch += __syncthreads_count(i < nnear && near_at(min(i, nnear - 1)) < prm.ncharged);
        }
        if (staged) stage(0, nnear);
    }
    // ---- runs of 8 along z: far sums from the lines, then (LEAF) the near atoms.  A column's
    // points go to two threads in turn, so that neighbours write neighbouring points.
    const int my = LEAF ? hi[1] - lo[1] + 1 : BOX_S, mx = LEAF ? hi[0] - lo[0] + 1 : BOX_S, mz = hi[2] - lo[2] + 1;
    const int nrun = 2 * mx * my;
    for (int c0 = 0; c0 < nrun; c0 += NT) {
        const int c = min(c0 + tid, nrun - 1);  // threads past the end repeat the last run and store nothing
        const int h = c & 1, xy = c >> 1, x = xy / my, y = xy - x * my;
        {
            float2 z[NC][4];
#pragma unroll
            for (int j = 0; j < BOX_N; j++) {
                const float2 w = bc(s_wy[y][j]);
#pragma unroll
                for (int k = 0; k < NC; k++) {
                    const float4 v0 = line[(k * BOX_S + x) * 16 + 2 * j], v1 = line[(k * BOX_S + x) * 16 + 2 * j + 1];
                    z[k][0] = j ? fma2(w, make_float2(v0.x, v0.y), z[k][0]) : mul2(w, make_float2(v0.x, v0.y));
                    z[k][1] = j ? fma2(w, make_float2(v0.z, v0.w), z[k][1]) : mul2(w, make_float2(v0.z, v0.w));
                    z[k][2] = j ? fma2(w, make_float2(v1.x, v1.y), z[k][2]) : mul2(w, make_float2(v1.x, v1.y));
                    z[k][3] = j ? fma2(w, make_float2(v1.z, v1.w), z[k][3]) : mul2(w, make_float2(v1.z, v1.w));
                }
            }
            S.zero();
#pragma unroll
            for (int j = 0; j < BOX_N; j++) {
                const float4 *wz = reinterpret_cast<const float4 *>(&s_wz[h][j][0]);
                const float4 w0 = wz[0], w1 = wz[1];
#pragma unroll
                for (int k = 0; k < NC; k++) {
                    const float2 f = bc((j & 1) ? z[k][j >> 1].y : z[k][j >> 1].x);
                    S.at(k, 0) = fma2(f, make_float2(w0.x, w0.y), S.at(k, 0));
                    S.at(k, 1) = fma2(f, make_float2(w0.z, w0.w), S.at(k, 1));
                    S.at(k, 2) = fma2(f, make_float2(w1.x, w1.y), S.at(k, 2));
                    S.at(k, 3) = fma2(f, make_float2(w1.z, w1.w), S.at(k, 3));
                }
            }
        }
        if constexpr (!LEAF) {
            // node column (x & 7, y & 7) of child (x >> 3, y >> 3, h)
            const int ch[3] = {2 * b[0] + (x >> 3), 2 * b[1] + (y >> 3), 2 * b[2] + h};
            if (!box_there(B, level - 1, ch)) continue;
            const BoxShare cs = box_share<NC>(prm, B, level - 1, ch);
            if (!share_has_slot<NC>(cs, level - 1)) continue;
#pragma unroll
            for (int k = 0; k < NC; k++)
#pragma unroll
                for (int e = 0; e < 2; e++)
                    *share_slot<NC>(cs, level - 1, k * (BOX_N3 / 4) + 2 * ((x & 7) * 8 + (y & 7)) + e) =
                        make_float4(S.at(k, 2 * e).x, S.at(k, 2 * e).y, S.at(k, 2 * e + 1).x, S.at(k, 2 * e + 1).y);
        } else {
            dfl o[3];
#pragma unroll
            for (int k = 0; k < 3; k++) o[k] = df_add(df_add(s_pt[0][x][k], s_pt[1][y][k]), s_pt[2][h][k]);
            // Two-level sums when there are many near atoms: BOX_FOLD of them join the running sums.
            float2 *run = reinterpret_cast<float2 *>(line + NC * BOX_S * 16);
            const bool fold = nnear > BOX_FOLD;
            auto join = [&](bool first) {
#pragma unroll
                for (int k = 0; k < Sums::NC1; k++)
#pragma unroll
                    for (int p = 0; p < BOX_P2; p++) {
                        float2 &r = run[(k * BOX_P2 + p) * NT + tid];
                        r = first ? S.at(k, p) : add2(r, S.at(k, p));
                    }
                S.a.zero();
            };
            if (fold) join(true);
            if (listed) {
                for (int n0 = 0; n0 < nnear; n0 += BOX_STAGE) {
                    const int n1 = min(nnear, n0 + BOX_STAGE);
                    if (!staged) stage(n0, n1);
                    for (int m0 = n0; m0 < n1; m0 += BOX_FOLD) {
                        const int m1 = min(n1, m0 + BOX_FOLD), mq = min(max(nch, m0), m1);
                        const float4 *T = tiles + 3 * (m0 - n0);
                        for (int j = m0; j < mq; j++, T += 3) box_add<MODE, WITH_E, ORTHO, true>(prm, B, o, nullptr, T[0], T[1], T[2], true, S);
                        if (MODE != M_COUL)
                            for (int j = mq; j < m1; j++, T += 3) box_add<MODE, WITH_E, ORTHO, true>(prm, B, o, nullptr, T[0], T[1], T[2], false, S);
                        if (fold) join(false);
                    }
                    if (!staged) __syncthreads();
                }
            } else {  // more near atoms than the list holds: through all atoms again
                for (int t = 0; t < ntiles; t++) {
                    const float4 *T = tiles + (t & 1) * NT * FF_REC;
                    gather(t, true);
                    pick(T, min(NT, nat - t * NT), 0, true);
                    __syncthreads();
                    for (int i = 0; i < nmid; i++) {
                        const int j = pk.mid[i];
                        const float4 r2r = T[3 * j + 2];
                        box_add<MODE, WITH_E, ORTHO, true>(prm, B, o, nullptr, T[3 * j], T[3 * j + 1], r2r, r2r.w != 0.f, S);
                    }
                    if (nmid > 0) join(false);
                    __syncthreads();
                }
            }
            if (fold) {
#pragma unroll
                for (int k = 0; k < Sums::NC1; k++)
#pragma unroll
                    for (int p = 0; p < BOX_P2; p++) S.at(k, p) = run[(k * BOX_P2 + p) * NT + tid];
            }
            if (c0 + tid >= nrun) continue;
            float4 *dst = prm.FE + ((long long)(lo[0] + x) * prm.ns[1] + lo[1] + y) * prm.ns[2] + lo[2] + h;
#pragma unroll
            for (int i = 0; i < 8; i++) {
                if (2 * i + h >= mz) break;
                const int p = i >> 1;
                float t[4], u[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    t[k] = k < Sums::NC1 ? ((i & 1) ? S.at(k, p).y : S.at(k, p).x) : 0.f;
                    if (MODE == M_LJC && k < Sums::NC1)
                        u[k] = (i & 1) ? S.at(Sums::NC1 + k, p).y : S.at(Sums::NC1 + k, p).x;
                }
                float4 f = finalize<MODE, WITH_E>(t[0], t[1], t[2], t[3], u[0], u[1], u[2], u[3], prm);
                if (!finite4(f)) {
                    // The displacement from the atom may be nothing but rounding: ff_block's.
                    double q[3];
#pragma unroll
                    for (int k = 0; k < 3; k++)
                        q[k] = ((prm.dA[k] * (prm.i0[0] + lo[0] + x)) + prm.dB[k] * (prm.i0[1] + lo[1] + y)) +
                               prm.dC[k] * (prm.i0[2] + lo[2] + 2 * i + h);
                    if (listed && staged) {
                        float far[8] = {};  // component k of the far sums, from the lines again
#pragma unroll 1
                        for (int k = 0; k < NC; k++) {
                            float v = 0.f;
#pragma unroll 1
                            for (int e = 0; e < 64; e++)
                                v = fmaf(s_wy[y][e >> 3] * s_wz[h][e & 7][i], reinterpret_cast<const float *>(line)[(k * BOX_S + x) * 64 + e], v);
                            far[k < Sums::NC1 ? k : k - Sums::NC1 + 4] = v;
                        }
                        f = box_point_slow<MODE, WITH_E>(prm, df_from(q[0]), df_from(q[1]), df_from(q[2]), tiles, nnear, nch,
                                                         make_float4(far[0], far[1], far[2], far[3]),
                                                         make_float4(far[4], far[5], far[6], far[7]));
                    } else {
                        f = point_slow<MODE, WITH_E>(prm, q[0], q[1], q[2]);
                    }
                }
                float4 *d = dst + 2 * i;
                if (prm.accumulate) {
                    const float4 old = *d;
                    f = make_float4(f.x + old.x, f.y + old.y, f.z + old.z, f.w + old.w);
                }
                *d = f;
            }
        }
    }
}

// ---------------------------------------------------------------------------- host

// One level.  Upper boxes in CTAs of 128 threads when there are more of them than two CTAs of 256 a
// SM: 343 boxes of 512 nodes and 342 atoms (a 200^3 grid) are then one wave of 152 SMs, not two.
template <int MODE, bool WITH_E, bool ORTHO, bool LEAF, int NT>
static int launch_box_level(const FFParams &prm, const BoxPrm &B, long long n, cudaStream_t st) {
    constexpr int smem = (int)box_smem<MODE, WITH_E, NT>();
    PPGPU_CUDA(cudaFuncSetAttribute(ff_box_kernel<MODE, WITH_E, ORTHO, LEAF, NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem),
               "ff_box shared memory");
    ff_box_kernel<MODE, WITH_E, ORTHO, LEAF, NT><<<(unsigned)n, NT, smem, st>>>(prm, B);
    PPGPU_CHECK_LAUNCH("ff_box_kernel launch");
    return PPGPU_OK;
}

template <int MODE, bool WITH_E, bool ORTHO>
static int launch_box(const FFParams &prm, BoxPrm B, cudaStream_t st) {
    for (B.level = B.levels; B.level >= 0; B.level--) {
        long long n = 1;
        for (int k = 0; k < 3; k++) n *= ((B.nb[k] - 1) >> B.level) + 1;
        if (n > 0x7fffffffLL) return set_error(PPGPU_ERR_ARG, "ff grid too large (%lld boxes)", n);
        int rc;
        if (B.level == 0)
            rc = launch_box_level<MODE, WITH_E, ORTHO, true, BOX_NT>(prm, B, n, st);
        else if (n > 304)
            rc = launch_box_level<MODE, WITH_E, ORTHO, false, 128>(prm, B, n, st);
        else
            rc = launch_box_level<MODE, WITH_E, ORTHO, false, 256>(prm, B, n, st);
        if (rc) return rc;
    }
    return set_ok();
}

template <int MODE>
static int launch_box_mode(const FFParams &prm, const BoxPrm &B, bool with_e, bool ortho, cudaStream_t st) {
    if (with_e) return ortho ? launch_box<MODE, true, true>(prm, B, st) : launch_box<MODE, true, false>(prm, B, st);
    return ortho ? launch_box<MODE, false, true>(prm, B, st) : launch_box<MODE, false, false>(prm, B, st);
}

// Largest distance of a tip charge from the probe's position.
static double tip_reach(const FFParams &prm) {
    double q = 0.0;
    for (int k = 0; k < prm.nqa; k++) q = std::max(q, (double)fabsf(prm.QZa[k]));
    return q;
}

// Grids and atoms summed by boxes.  Measured on a GB300, ff_block -> boxes (LJ + Coulomb, all atoms
// charged, 0.05 to 0.3 A steps alike):
//   200^3 points,   342 atoms          1.40 -> 0.28 ms     400x400x250, 18540 atoms  270 -> 8.1 ms,
//                                                          800x800x500                2120 -> 16.8 ms
//   128^3 (512 leaves): 540 atoms      0.61 -> 0.21 ms,  90: 0.113 -> 0.060,  60: 0.083 -> 0.077, 20: 0.041 -> 0.050
//   220^3 (2744 leaves): 90 atoms      0.51 -> 0.20 ms,  60: 0.36 -> 0.22,    20: 0.15 -> 0.165
//   64^3 (64 leaves), 540 atoms        0.108 -> 0.152 ms: too few boxes to fill 152 SMs
//   AFMulator tip, 256x256x192:        38 atoms 1.05 -> 0.48 ms, 10 atoms 0.33 -> 0.23
// A box costs some 10 pairs a point whatever its atoms (classifying, interpolating, writing), which
// the far atoms have to save; a pair with the tip's charges counts for five.  With leaves of half
// diagonal H over 5 A nearly every atom within 35 A is near.
bool ff_box_rule(const FFParams &prm, int mode, int *levels) {
    BoxPrm B;
    double H;
    box_plan(prm, BOX_KAPPA, tip_reach(prm), &B, &H);
    const double boxes = (double)B.nb[0] * B.nb[1] * B.nb[2];
    const double nat = mode == M_COUL ? prm.ncharged : prm.natoms;
    const double pairs = nat + (mode == M_QZS && prm.nqa > 0 ? 4.0 * prm.ncharged : 0.0);
    // levels: 220^3, 342 atoms 0.43, 0.30, 0.32 ms with 0, 1, 2 (9.4e5 atom-boxes); 128^3, 540 atoms
    // 0.210, 0.217 (2.8e5); slab on 400x400x250 40, 12.3, 8.1 ms (1.9e8), on 240x240x150 14.2, 9.4, 9.4 (4.2e7)
    const double work = nat * boxes;
    *levels = work < 4e5 ? 0 : (work < 1e8 ? 1 : (work < 1e9 ? 2 : 3));
    return boxes >= 304 && H <= 5.0 && pairs >= 40.0 + 20480.0 / boxes;
}

int launch_ff_box(const FFParams &prm, int mode, bool with_e, bool ortho, int levels, cudaStream_t st) {
    BoxPrm B;
    double H;
    box_plan(prm, BOX_KAPPA, tip_reach(prm), &B, &H);
    B.levels = prm.accumulate ? 0 : std::min(levels, BOX_LEVELS);
    switch (mode) {
        case M_LJ:
            return launch_box_mode<M_LJ>(prm, B, with_e, ortho, st);
        case M_COUL:
            return launch_box_mode<M_COUL>(prm, B, with_e, ortho, st);
        case M_LJC:
            return launch_box_mode<M_LJC>(prm, B, with_e, ortho, st);
        default:
            return launch_box_mode<M_QZS>(prm, B, with_e, ortho, st);
    }
}

}  // namespace ppgpu
