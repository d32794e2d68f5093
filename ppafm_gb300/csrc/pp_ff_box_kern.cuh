// pp_ff_box_kern.cuh -- force-field grids by boxes: near atoms point by point, far atoms on
// Chebyshev nodes.
//
// The field of an atom that is far from a box of grid points is smooth over the box, so it is
// summed on a few nodes and interpolated from there, instead of being summed at every point
// (the one-level form of the kernel-independent, interpolation-based fast summation: W. Fong and
// E. Darve, "The black-box fast multipole method", J. Comput. Phys. 228 (2009)).  The sums are
// those of ff_block (pp_ff_dev.cuh): the same pair interactions, in the same arithmetic.
//
//  * A leaf box is up to 16 x 16 x 16 points, one CTA.  Its far atoms are summed on N^3 Chebyshev
//    nodes (N = 8 or 10: 512 or 1000 against 4096 points), its near ones at the points.
//  * Levels above it: boxes of 2 x 2 x 2 boxes of the level below, with the same N^3 nodes, so
//    that atoms farther away cost 1/8 at each level.  An atom is summed at the highest level at
//    which it is far from the leaf's ancestor.  An upper box interpolates its nodes' sums to the
//    nodes of its 8 children, which start from them.
//  * Far at a level: R >= kappa H from the box's centre, H its half diagonal; kappa 7 with 8 nodes,
//    4.25 with 10.  The interpolation error of the r^-7 force (dispersion, the steepest that
//    matters at that distance) is then below 1.5e-7 of the pair's force, under the ~4e-7 rounding
//    of a float32 pair term.  The r^-13 repulsion needs more distance the stronger it is beside the
//    dispersion: an atom whose coefficients do not satisfy the bound in `box_far` stays near,
//    whatever they are.
//  * What is handed to a child lies in the child's own part of the output grid until its CTAs read
//    it and later write their own there: no workspace.  A box that is too small to hold it (a
//    remainder at the grid's edge), and every box when FE is accumulated into, sums its far
//    atoms itself.
//
// Bound by the issue of float32 instructions like ff_block, on far fewer pairs.  Figures beside
// box_choice (pp_ff_box.cu).
#pragma once

#include "pp_ff_box_dev.cuh"

namespace ppgpu {

constexpr int BOX_FOLD = 64;     // near atoms summed before they join a point's running sum
constexpr int BOX_P2 = 4;        // pairs of a thread's run of 8 points along z (of nodes: P2N)

// --------------------------------------------------------------------------- sums

template <int MODE, bool WITH_E, int P2>
struct BoxSums {
    static constexpr int U = (MODE == M_LJC) ? P2 : 1;
    static constexpr int NC1 = WITH_E ? 4 : 3;                   // components of one sum
    static constexpr int NC = (MODE == M_LJC) ? 2 * NC1 : NC1;   // LJC: LJ, then electrostatic
    Acc<P2> a;
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

// Adds one atom to the sums of a thread's run of positions: the double-float position o and offsets
// from it, as floats (nodes: off[axis][i], one after another, in shared memory) or in two parts (POINT: B.offh, offl).
// Points can be close to the atom, where the rounding of their offsets would count.
template <int MODE, bool WITH_E, bool ORTHO, bool POINT, int P2>
__device__ __forceinline__ void box_add(const FFParams &prm, const BoxPrm &B, const dfl o[3], const float *off,
                                        const float4 &r0, const float4 &r1, const float4 &r2r, bool charged,
                                        BoxSums<MODE, WITH_E, P2> &S) {
    const float eps = prm.eps;
    float h[3] = {o[0].h + r0.x, o[1].h + r0.y, o[2].h + r1.x}, l[3] = {o[0].l + r0.z, o[1].l + r0.w, o[2].l + r1.y};
    if (POINT) {  // what the run's middle less the atom loses would count where a point's offset cancels it
        const float a[3] = {r0.x, r0.y, r1.x};
#pragma unroll
        for (int k = ORTHO ? 2 : 0; k < 3; k++) l[k] += two_sum(o[k].h, a[k]).l;
    }
    const float2 c6n6 = bc(r1.z), c12x12 = bc(r1.w), c6n = bc(r2r.x), c12 = bc(r2r.y), kqq = bc(r2r.z);
    const float x0 = h[0] + l[0], y0 = h[1] + l[1], z0 = h[2] + l[2];
    const float2 xy0 = bc(fmaf(x0, x0, fmaf(y0, y0, eps)));
    auto along = [&](int k, float v0, int p) -> float2 {  // component k of pair p's displacement
        if constexpr (POINT)
            return add2(add2(bc(h[k]), make_float2(B.offh[k][2 * p], B.offh[k][2 * p + 1])),
                        add2(bc(l[k]), make_float2(B.offl[k][2 * p], B.offl[k][2 * p + 1])));
        else
            return add2(bc(v0), make_float2(off[2 * P2 * k + 2 * p], off[2 * P2 * k + 2 * p + 1]));
    };
#pragma unroll
    for (int p = 0; p < P2; p++) {
        const float2 dz = along(2, z0, p);
        const float2 dx = ORTHO ? bc(x0) : along(0, x0, p), dy = ORTHO ? bc(y0) : along(1, y0, p);
        const float2 xy = ORTHO ? xy0 : fma2(dy, dy, fma2(dx, dx, bc(eps)));
        const float2 r2 = fma2(dz, dz, xy);
        if constexpr (MODE == M_COUL) {
            const float2 ir = rsqrt2(r2);
            coul_ir<WITH_E, P2>(ir, mul2(ir, ir), dx, dy, dz, kqq, S.a, p);
        } else if constexpr (MODE == M_LJC) {
            if (charged)
                ljc_ir<WITH_E, P2>(rsqrt2(r2), dx, dy, dz, c6n6, c12x12, c6n, c12, kqq, S.a, S.u, p);
            else
                lj_ir2<WITH_E, P2>(rcp2(r2), dx, dy, dz, c6n6, c12x12, c6n, c12, S.a, p);
        } else {
            lj_ir2<WITH_E, P2>(rcp2(r2), dx, dy, dz, c6n6, c12x12, c6n, c12, S.a, p);
            if (MODE == M_QZS && charged) qzs_tip<WITH_E, P2>(prm, r2r.z, r2, dx, dy, dz, xy, S.a, p);
        }
    }
}

// Rare: a point whose float32 sums overflow, within ~5e-3 A of an atom: the far sums t (and u) and
// the listed near atoms (charged ones first) with r^2 floored like ff_block's slow path.
template <int MODE, bool WITH_E>
__device__ __noinline__ float4 box_point_slow(const FFParams &prm, dfl x, dfl y, dfl z, const BoxNear &list, bool wide, int nnear,
                                              int ncharged, float4 t, float4 u) {
    for (int j = 0; j < nnear; j++) {
        const float4 *a = prm.atoms + (size_t)list.at(wide, j) * FF_REC;
        const float4 r0 = ldg4(a), r1 = ldg4(a + 1), r2r = ldg4(a + 2);
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
            float4 &f = MODE == M_LJC ? u : t;
            f.x = fmaf(fq, dx, f.x);
            f.y = fmaf(fq, dy, f.y);
            f.z = fmaf(fq, dq, f.z);
            f.w += eq;
        }
    }
    return finalize<MODE, WITH_E>(t.x, t.y, t.z, t.w, u.x, u.y, u.z, u.w, prm);
}

// ------------------------------------------------------------------------- the kernel

// Threads of a CTA and the node columns: each thread has a column and one of SUBS parts of the atoms
// (N = 8: 4 parts of 64 columns, N = 10: 2 of 100, in 7 of the 8 warps).  Their sums join running sums over
// the tiles (two-level summation) in shared memory: those of the even parts, then, after the
// threads have met, those of the odd ones.  Sums of the nodes are laid out [component][pair along
// z][x][y], wherever they are: free of bank conflicts for the threads' columns, and two
// neighbours along y in one load.
template <int N>
struct BoxCols {
    static constexpr int N2 = N * N, N3 = N2 * N, P2 = N / 2, SUBS = BOX_NT / N2, ACC = SUBS / 2;
};
template <int N, class Sums>
__device__ __forceinline__ void box_join(Sums &M, float2 *nodes, int sub, int col, int odd) {
    using C = BoxCols<N>;
    if (sub >= C::SUBS || (sub & 1) != odd) return;
#pragma unroll
    for (int k = 0; k < Sums::NC; k++)
#pragma unroll
        for (int p = 0; p < C::P2; p++) {
            float2 &r = nodes[(((sub >> 1) * Sums::NC + k) * C::P2 + p) * C::N2 + col];
            r = add2(r, M.at(k, p));
        }
    M.zero();
}

// Positions of the nodes: middles of the columns (z: the middle only), offsets along them.
template <int N>
__device__ __forceinline__ void box_node_table(const FFParams &prm, const BoxPrm &B, int level, const int b[3], int i,
                                               dfl (*node)[N][3], float (*off)[N]) {
    const int a = i / N, n = i % N;
    int l, h;
    box_span(prm, B, level, a, a == 0 ? b[0] : (a == 1 ? b[1] : b[2]), l, h);
    const float mid = 0.5f * (float)(l + h) + (float)prm.i0[a];
    const dfl e = df_mul_f(cheb_t<N>(n), box_half(l, h)), g = a < 2 ? df_add(e, {mid, 0.f}) : dfl{mid, 0.f};  // middle + half t_n, in steps
#pragma unroll
    for (int k = 0; k < 3; k++) {
        node[a][n][k] = df_mul(B.step[a][k], g);
        if (a == 2) off[k][n] = df_round(df_mul(B.step[2][k], e));
    }
}

// ---------------------------------------------------------------------- upper boxes
//
// A cluster of 1 to 8 CTAs a box: each sums a part of the atoms on the nodes, adds up what all of
// them have, and interpolates to some of the children, along z, y and x.  Atoms and children are
// few where the boxes are many and many where they are few (the top level of the slab: 32 boxes
// of 10 000 atoms), so that one CTA a box left most of the SMs idle.

template <int MODE, bool WITH_E, int N>
struct BoxUpSmem {  // the atom tiles, then the sums along z; this CTA's sums, then those along y; the box's sums
    static constexpr int NC = BoxSums<MODE, WITH_E, 1>::NC;
    static constexpr size_t tiles = sizeof(float4) * 2 * BOX_NT * FF_REC, nodes = sizeof(float) * NC * N * N * N;
    static constexpr size_t own = tiles > nodes ? tiles : nodes, sum = own + BoxCols<N>::ACC * nodes, size = sum + nodes;
};

template <int MODE, bool WITH_E, bool ORTHO, int N>
__global__ void __launch_bounds__(BOX_NT, 2) box_up_kernel(const __grid_constant__ FFParams prm, const __grid_constant__ BoxPrm B) {
    using Smem = BoxUpSmem<MODE, WITH_E, N>;
    using Cols = BoxCols<N>;
    constexpr int NC = Smem::NC, NT = BOX_NT, N2 = Cols::N2, N3 = Cols::N3, P2N = Cols::P2, SUBS = Cols::SUBS, C4 = NC * N3 / 4;
    extern __shared__ __align__(128) unsigned char box_raw[];
    float4 *tiles = reinterpret_cast<float4 *>(box_raw);
    float4 *own = reinterpret_cast<float4 *>(box_raw + Smem::own), *sum = reinterpret_cast<float4 *>(box_raw + Smem::sum);
    __shared__ unsigned short s_left[BOX_LEFT];
    __shared__ BoxPick<NT> pk;
    __shared__ int s_idx[2][NT], s_count;
    __shared__ dfl s_node[3][N][3];
    __shared__ float s_off[3][N];
    __shared__ __align__(16) float s_w[3][2][N][12];  // [axis][child][node of the box][node of the child]

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int level = B.level, rank = cluster_rank(), ncta = cluster_size();
    const int nat = (MODE == M_COUL) ? prm.ncharged : prm.natoms;
    int b[3], lo[3], hi[3];
    box_of_cta(prm, B, level, blockIdx.x / ncta, b, lo, hi);
    BoxShare share;
    bool handed = false;  // the parent's sums are there
    int nlist = -1;       // atoms that the parent left to this box (-1: no list)
    if (level < B.levels) {
        share = box_share<N, NC>(prm, B, level, b);
        handed = share_has_sums<N, NC>(share);
        if (handed && share.room > 0) nlist = *share_count<N, NC>(share);
    }
    const int nanc = handed ? B.levels - level : 0;
    const int ncand = nlist >= 0 ? nlist : nat, per = (ncand + ncta - 1) / ncta;
    const int first = min(rank * per, ncand), last = min(first + per, ncand), ntiles = (last - first + NT - 1) / NT;
    auto index = [&](int t) -> int {  // this thread's atom of tile t
        const int i = first + t * NT + tid;
        return i < last ? (nlist >= 0 ? (int)*share_list<N, NC>(share, i) : i) : -1;
    };
    auto fetch = [&](int t, int j) {
        if (j >= 0) {
            const float4 *a = prm.atoms + (size_t)j * FF_REC;
            float4 *d = tiles + ((t & 1) * NT + tid) * FF_REC;
#pragma unroll
            for (int k = 0; k < FF_REC; k++) async_copy16(d + k, a + k);
            s_idx[t & 1][tid] = j;
        }
        async_commit();
    };
    int j0 = index(0), j1 = index(1);
    fetch(0, j0);
    if (warp == 1 && lane <= nanc) pk.centre[lane] = box_centre(prm, B, level, b, lane);
    if (warp == 0 && lane < 3 * N) box_node_table<N>(prm, B, level, b, lane, s_node, s_off);
    for (int i = tid; i < Cols::ACC * C4; i += NT) own[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    __syncthreads();
    auto weights = [&]() {  // by the last warp, which has no node columns with 10 nodes
        for (int i = lane; i < 6 * N; i += 32) {
            const int a = i / (2 * N), c = i / N % 2, n = i % N;
            dfl x;
            if (box_child_node<N>(prm, B, level, a, a == 0 ? b[0] : (a == 1 ? b[1] : b[2]), c, n, x))
                cheb_row<N>(x, [&](int k, dfl w) { s_w[a][c][k][n] = df_round(w); });
        }
    };
    // ---- far atoms on the nodes: thread = node column (ia, ib), one of SUBS parts of the atoms
    const int sub = tid / N2, col = tid % N2;
    BoxSums<MODE, WITH_E, P2N> M;
    M.zero();
    dfl on[3];
#pragma unroll
    for (int k = 0; k < 3; k++) on[k] = df_add(df_add(s_node[0][col / N][k], s_node[1][col % N][k]), s_node[2][0][k]);
    int nmid = 0, nzero = 0, place = -1, nleft = 0;
    for (int t = 0; t < ntiles; t++) {
        const float4 *T = tiles + (t & 1) * NT * FF_REC;
        const int j = j0;
        j0 = j1;
        j1 = index(t + 2);
        fetch(t + 1, j0);
        async_wait<1>();
        box_pick<MODE, N, NT>(B, pk, level, nanc, T, min(NT, last - first - t * NT), 1, true, nmid, nzero, place);
        if (place >= 0 && nleft + place < BOX_LEFT) s_left[nleft + place] = (unsigned short)j;
        nleft += nzero;
        __syncthreads();
        if (t == 0 && warp == NT / 32 - 1) weights();
        if (sub < SUBS) {
            for (int i = sub; i < nmid; i += SUBS) {
                const int q = pk.mid[i];
                box_add<MODE, WITH_E, ORTHO, false>(prm, B, on, &s_off[0][0], T[3 * q], T[3 * q + 1], T[3 * q + 2], s_idx[t & 1][q] < prm.ncharged, M);
            }
        }
        box_join<N>(M, reinterpret_cast<float2 *>(own), sub, col, 0);
        __syncthreads();
        box_join<N>(M, reinterpret_cast<float2 *>(own), sub, col, 1);
    }
    async_wait<0>();
    if (Cols::ACC == 2) {
        __syncthreads();
        for (int i = tid; i < C4; i += NT) {
            const float4 u = own[i], v = own[C4 + i];
            own[i] = make_float4(u.x + v.x, u.y + v.y, u.z + v.z, u.w + v.w);
        }
    }
    if (ntiles == 0 && warp == NT / 32 - 1) weights();
    if (tid == 0) s_count = prm.natoms <= 65536 && nleft <= BOX_LEFT ? nleft : -1;
    // ---- the box's sums: of all CTAs in turn and the parent's interpolated ones
    cluster_meet();
    int before = 0, all = 0;
    for (int q = 0; q < ncta; q++) {
        const int n = cluster_ldi(cluster_addr(&s_count, q));
        if (q < rank) before += n;
        all = n < 0 || all < 0 ? -1 : all + n;
    }
    for (int i = tid; i < C4; i += NT) {
        float4 v = handed ? *share_cell(share, i) : make_float4(0.f, 0.f, 0.f, 0.f);
        for (int q = 0; q < ncta; q++) {
            const float4 o = cluster_ld4(cluster_addr(own + i, q));
            v = make_float4(v.x + o.x, v.y + o.y, v.z + o.z, v.w + o.w);
        }
        sum[i] = v;
    }
    cluster_meet();  // all CTAs have read the box's part of the grid, and this one's sums
    box_leave<N, NC, NT>(prm, B, level, b, s_left, nleft, before, all, rank == 0);
    float2 *lz = reinterpret_cast<float2 *>(tiles), *ly = reinterpret_cast<float2 *>(own);
    for (int q = rank; q < 8; q += ncta) {
        const int c[3] = {q >> 2, (q >> 1) & 1, q & 1}, ch[3] = {2 * b[0] + c[0], 2 * b[1] + c[1], 2 * b[2] + c[2]};
        if (!box_there(B, level - 1, ch)) continue;
        const BoxShare cs = box_share<N, NC>(prm, B, level - 1, ch);
        if (!share_has_sums<N, NC>(cs)) continue;
        // ---- along z: a column of nodes a thread
        for (int i = tid; i < NC * N2; i += NT) {
            const int k = i / N2, e = k * (P2N * N2) + i - k * N2;
            const float2 *v = reinterpret_cast<const float2 *>(sum) + e;
            float2 s[P2N];
#pragma unroll
            for (int c2 = 0; c2 < P2N; c2++) {
                const float2 f = v[c2 * N2], f0 = bc(f.x), f1 = bc(f.y);
                const float2 *w0 = reinterpret_cast<const float2 *>(s_w[2][c[2]][2 * c2]), *w1 = reinterpret_cast<const float2 *>(s_w[2][c[2]][2 * c2 + 1]);
#pragma unroll
                for (int p = 0; p < P2N; p++) s[p] = fma2(f1, w1[p], c2 ? fma2(f0, w0[p], s[p]) : mul2(f0, w0[p]));
            }
#pragma unroll
            for (int p = 0; p < P2N; p++) lz[e + p * N2] = s[p];
        }
        __syncthreads();
        // ---- along y: a column of the child's nodes
        for (int i = tid; i < NC * N2; i += NT) {
            const int k = i / N2, xy = i - k * N2, x = xy / N, y = xy - x * N;
            float2 s[P2N];
#pragma unroll
            for (int j = 0; j < N; j += 2) {
                const float2 w0 = bc(s_w[1][c[1]][j][y]), w1 = bc(s_w[1][c[1]][j + 1][y]);
#pragma unroll
                for (int p = 0; p < P2N; p++) {
                    const float4 f = reinterpret_cast<const float4 *>(lz)[(((k * P2N + p) * N + x) * N + j) >> 1];
                    s[p] = fma2(w1, make_float2(f.z, f.w), j ? fma2(w0, make_float2(f.x, f.y), s[p]) : mul2(w0, make_float2(f.x, f.y)));
                }
            }
#pragma unroll
            for (int p = 0; p < P2N; p++) ly[(k * P2N + p) * N2 + xy] = s[p];
        }
        __syncthreads();
        // ---- along x: pairs of nodes of two columns
        for (int i = tid; i < C4; i += NT) {
            const int kp = i / (N2 / 2), r = i - kp * (N2 / 2), x = r / (N / 2), y2 = r - x * (N / 2);
            float2 s0, s1;
#pragma unroll
            for (int a = 0; a < N; a++) {
                const float2 w = bc(s_w[0][c[0]][a][x]);
                const float4 v = reinterpret_cast<const float4 *>(ly)[(kp * N + a) * (N / 2) + y2];
                s0 = a ? fma2(w, make_float2(v.x, v.y), s0) : mul2(w, make_float2(v.x, v.y));
                s1 = a ? fma2(w, make_float2(v.z, v.w), s1) : mul2(w, make_float2(v.z, v.w));
            }
            *share_cell(cs, i) = make_float4(s0.x, s0.y, s1.x, s1.y);
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------- leaves

// Shared memory: two atom tiles, then the sums interpolated along x; behind them the nodes' sums, then
// near atoms and the points' running sums.
template <int MODE, bool WITH_E, int N>
struct BoxSmem {
    static constexpr int NC1 = WITH_E ? 4 : 3, NC = MODE == M_LJC ? 2 * NC1 : NC1;
    static constexpr size_t cmax(size_t a, size_t b) { return a > b ? a : b; }
    static constexpr size_t nodes = cmax(sizeof(float4) * 2 * BOX_NT * FF_REC, sizeof(float) * NC * BOX_S * N * N);
    static constexpr size_t run = nodes + sizeof(float4) * BOX_STAGE * FF_REC;
    static constexpr size_t size = cmax(nodes + sizeof(float) * BoxCols<N>::ACC * NC * N * N * N, run + sizeof(float2) * NC1 * BOX_P2 * BOX_NT);
};

// CTAs of 256 threads: the warps of a scheduler then run the same part of the long straight-line code
// (with 128, four CTAs at four places waited on instruction fetches), two CTAs a SM at 128
// registers.
template <int MODE, bool WITH_E, bool ORTHO, int N>
__global__ void __launch_bounds__(BOX_NT, 2) ff_box_kernel(const __grid_constant__ FFParams prm, const __grid_constant__ BoxPrm B) {
    using Smem = BoxSmem<MODE, WITH_E, N>;
    using Cols = BoxCols<N>;
    constexpr int NC = Smem::NC, NC1 = Smem::NC1, NT = BOX_NT, N2 = Cols::N2, N3 = Cols::N3, P2N = Cols::P2, SUBS = Cols::SUBS;
    constexpr int C4 = NC * N3 / 4, level = 0;
    extern __shared__ __align__(128) unsigned char box_raw[];
    float4 *tiles = reinterpret_cast<float4 *>(box_raw), *line = tiles;
    float4 *nodes = reinterpret_cast<float4 *>(box_raw + Smem::nodes), *near = nodes;
    __shared__ uint64_t bar[2];
    __shared__ BoxNear s_near;
    __shared__ BoxPick<NT> pk;
    __shared__ dfl s_node[3][N][3];
    __shared__ float s_off[3][N];
    __shared__ dfl s_pt[3][BOX_S][3];  // parts of the points' positions, runs along z from their middle
    __shared__ __align__(16) float s_wx[BOX_S][N], s_wy[BOX_S][N];
    __shared__ __align__(16) float s_wz[2][N][8];  // [half of a column][node][point]

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nat = (MODE == M_COUL) ? prm.ncharged : prm.natoms;
    const int ntiles = (nat + NT - 1) / NT;
    int b[3], lo[3], hi[3];
    box_of_cta(prm, B, level, blockIdx.x, b, lo, hi);
    BoxShare share;
    bool handed = false;  // the parent's sums are there
    int nlist = -1;       // atoms that the parent left to this box (-1: no list)
    if (level < B.levels) {
        share = box_share<N, NC>(prm, B, level, b);
        handed = share_has_sums<N, NC>(share);
        if (handed && share.room > 0) nlist = *share_count<N, NC>(share);
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
    if (warp == 0 && lane < 3 * N) box_node_table<N>(prm, B, level, b, lane, s_node, s_off);
    if (warp >= 2 && warp < 4 && tid - 64 < 34) {
        const int i = tid - 64, a = i >> 4, j = i & 15;
        const float g = (float)(prm.i0[a] + (a == 0 ? lo[0] : (a == 1 ? lo[1] : lo[2])) + j) + (a == 2 ? 7.f : 0.f);
#pragma unroll
        for (int k = 0; k < 3; k++) s_pt[a][j][k] = df_mul_f(B.step[a][k], g);
    }
    for (int i = tid; i < BOX_S * N; i += NT) {
        const int pt = i / N, k = i % N;
        s_wx[pt][k] = cheb_points<N>().w[hi[0] - lo[0] + 1][pt][k];
        s_wy[pt][k] = cheb_points<N>().w[hi[1] - lo[1] + 1][pt][k];
        s_wz[pt & 1][k][pt >> 1] = cheb_points<N>().w[hi[2] - lo[2] + 1][pt][k];
    }
    for (int i = tid; i < C4; i += NT) {  // the parent's sums
        if (handed) async_copy16(nodes + i, share_cell(share, i));
        else nodes[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (Cols::ACC == 2) nodes[C4 + i] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    async_commit();
    // ---- far atoms on the nodes, as in box_up_kernel
    const int sub = tid / N2, col = tid % N2;
    BoxSums<MODE, WITH_E, P2N> M;
    M.zero();
    async_wait<0>();
    __syncthreads();
    dfl on[3];
#pragma unroll
    for (int k = 0; k < 3; k++) on[k] = df_add(df_add(s_node[0][col / N][k], s_node[1][col % N][k]), s_node[2][0][k]);
    const bool wide = nat > 65536;  // near indices as int
    const int near_cap = wide ? BOX_NEAR / 2 : BOX_NEAR;
    auto near_at = [&](int i) -> int { return s_near.at(wide, i); };
    int nmid = 0, nzero = 0, place = -1;
    auto pick = [&](const float4 *T, int nj, int want, bool ok) {
        return box_pick<MODE, N, NT>(B, pk, level, nanc, T, nj, want, ok, nmid, nzero, place);
    };
    // This thread's atom of tile t of the parent's list, or (all) of all atoms, into the tile.  The
    // list is gone once the box writes its points.
    auto gather = [&](int t, bool all) -> int {
        const int i = t * NT + tid;
        int j = -1;
        if (i < (all ? nat : ncand)) {
            j = all ? i : (int)*share_list<N, NC>(share, i);
            box_gather(prm, (all ? near : tiles + (t & 1) * NT * FF_REC) + tid * FF_REC, j);
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
        if (place >= 0 && nnear + place < near_cap) s_near.set(wide, nnear + place, j0);
        nnear += nzero;
        __syncthreads();
        if (sub < SUBS) {
            for (int i = sub; i < nmid; i += SUBS) {
                const int j = pk.mid[i];
                const float4 r2r = T[3 * j + 2];
                const bool charged = nlist >= 0 ? r2r.w != 0.f : base + j < prm.ncharged;
                box_add<MODE, WITH_E, ORTHO, false>(prm, B, on, &s_off[0][0], T[3 * j], T[3 * j + 1], r2r, charged, M);
            }
        }
        box_join<N>(M, reinterpret_cast<float2 *>(nodes), sub, col, 0);
        __syncthreads();
        if (nlist < 0 && tid == 0 && t + 2 < ntiles) fetch(t + 2);
        box_join<N>(M, reinterpret_cast<float2 *>(nodes), sub, col, 1);
    }
    __syncthreads();
    // ---- interpolated along x: line[k][x][pair along z][y]
    constexpr int L4 = N2 / 4, XS = BOX_S, XG = XS / 4;  // a thread takes four nodes and every XG-th x
    for (int i = tid; i < NC * L4 * XG; i += NT) {
        const int x0 = i / (NC * L4), r = i - x0 * (NC * L4), kp = r / (N / 2), y2 = r - kp * (N / 2);
        const int k = kp / P2N, p = kp - k * P2N;
        float4 v[N];
#pragma unroll
        for (int a = 0; a < N; a++) {
            v[a] = nodes[(kp * N + a) * (N / 2) + y2];
            if (Cols::ACC == 2) {
                const float4 u = nodes[C4 + (kp * N + a) * (N / 2) + y2];
                v[a] = make_float4(v[a].x + u.x, v[a].y + u.y, v[a].z + u.z, v[a].w + u.w);
            }
        }
#pragma unroll 2
        for (int x = x0; x < XS; x += XG) {
            float2 s0 = make_float2(0.f, 0.f), s1 = s0;
#pragma unroll
            for (int a = 0; a < N; a++) {
                const float2 w = bc(s_wx[x][a]);
                s0 = fma2(w, make_float2(v[a].x, v[a].y), s0);
                s1 = fma2(w, make_float2(v[a].z, v[a].w), s1);
            }
            line[((k * XS + x) * P2N + p) * (N / 2) + y2] = make_float4(s0.x, s0.y, s1.x, s1.y);
        }
    }
    __syncthreads();
    // Components k0..k0+NK-1 along y at column (x, y): pairs of the nodes along z.
    auto along_y = [&](auto &z, int k0, int x, int y) {
        constexpr int NK = sizeof(z) / sizeof(z[0]);
#pragma unroll
        for (int j = 0; j < N; j += 2) {
            const float2 wj = *reinterpret_cast<const float2 *>(&s_wy[y][j]), w0 = bc(wj.x), w1 = bc(wj.y);
#pragma unroll
            for (int k = 0; k < NK; k++) {
                const float4 *v = line + ((k0 + k) * XS + x) * L4 + j / 2;
#pragma unroll
                for (int p = 0; p < P2N; p++) {
                    const float4 f = v[p * (N / 2)];  // two rows
                    z[k][p] = fma2(w1, make_float2(f.z, f.w), j ? fma2(w0, make_float2(f.x, f.y), z[k][p]) : mul2(w0, make_float2(f.x, f.y)));
                }
            }
        }
    };
    // Near atoms first..last-1 of the list into the tiles' space (the nodes' sums are done with).
    auto stage = [&](int first, int last) {
        for (int i = tid; i < (last - first) * FF_REC; i += NT)
            near[i] = ldg4(prm.atoms + (size_t)near_at(first + i / FF_REC) * FF_REC + i % FF_REC);
        __syncthreads();
    };
    const bool listed = nnear <= near_cap, staged = nnear <= BOX_STAGE;
    if (listed) {
        for (int i0 = 0; i0 < nnear; i0 += NT) {  // the charged ones come first
            const int i = i0 + tid;
            nch += __syncthreads_count(i < nnear && near_at(min(i, nnear - 1)) < prm.ncharged);
        }
        if (staged) stage(0, nnear);
    }
    // ---- runs of 8 along z: far sums from the lines, then the near atoms.  A column's
    // points go to two threads in turn, so that neighbours write neighbouring points.
    {
        const int my = hi[1] - lo[1] + 1, mx = hi[0] - lo[0] + 1, mz = hi[2] - lo[2] + 1;
        const int nrun = 2 * mx * my;
        for (int c0 = 0; c0 < nrun; c0 += NT) {
            const int c = min(c0 + tid, nrun - 1);  // threads past the end repeat the last run and store nothing
            const int h = c & 1, xy = c >> 1, x = xy / my, y = xy - x * my;
            BoxSums<MODE, WITH_E, BOX_P2> S;
            S.zero();
#pragma unroll
            for (int g = 0; g < NC; g += NC1) {
                float2 z[NC1][P2N];
                along_y(z, g, x, y);
#pragma unroll
                for (int j = 0; j < N; j++) {
                    const float4 *wz = reinterpret_cast<const float4 *>(&s_wz[h][j][0]);
                    const float4 w0 = wz[0], w1 = wz[1];
#pragma unroll
                    for (int k = 0; k < NC1; k++) {
                        const float2 f = bc((j & 1) ? z[k][j >> 1].y : z[k][j >> 1].x);
                        S.at(g + k, 0) = fma2(f, make_float2(w0.x, w0.y), S.at(g + k, 0));
                        S.at(g + k, 1) = fma2(f, make_float2(w0.z, w0.w), S.at(g + k, 1));
                        S.at(g + k, 2) = fma2(f, make_float2(w1.x, w1.y), S.at(g + k, 2));
                        S.at(g + k, 3) = fma2(f, make_float2(w1.z, w1.w), S.at(g + k, 3));
                    }
                }
            }
            dfl o[3];
#pragma unroll
            for (int k = 0; k < 3; k++) o[k] = df_add(df_add(s_pt[0][x][k], s_pt[1][y][k]), s_pt[2][h][k]);
            // Two-level sums when there are many near atoms: BOX_FOLD of them join the running sums.
            float2 *run = reinterpret_cast<float2 *>(box_raw + Smem::run);
            const bool fold = nnear > BOX_FOLD;
            auto join = [&](bool first) {
#pragma unroll
                for (int k = 0; k < NC1; k++)
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
                        const float4 *T = near + 3 * (m0 - n0);
                        for (int j = m0; j < mq; j++, T += 3) box_add<MODE, WITH_E, ORTHO, true>(prm, B, o, nullptr, T[0], T[1], T[2], true, S);
                        if (MODE != M_COUL)
                            for (int j = mq; j < m1; j++, T += 3) box_add<MODE, WITH_E, ORTHO, true>(prm, B, o, nullptr, T[0], T[1], T[2], false, S);
                        if (fold) join(false);
                    }
                    if (!staged) __syncthreads();
                }
            } else {  // more near atoms than the list holds: through all atoms again
                for (int t = 0; t < ntiles; t++) {
                    const float4 *T = near;
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
                for (int k = 0; k < NC1; k++)
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
                    t[k] = k < NC1 ? ((i & 1) ? S.at(k, p).y : S.at(k, p).x) : 0.f;
                    if (MODE == M_LJC && k < NC1)
                        u[k] = (i & 1) ? S.at(NC1 + k, p).y : S.at(NC1 + k, p).x;
                }
                float4 f = finalize<MODE, WITH_E>(t[0], t[1], t[2], t[3], u[0], u[1], u[2], u[3], prm);
                if (!finite4(f)) {
                    // The displacement from the atom may be nothing but rounding: ff_block's.
                    double q[3];
#pragma unroll
                    for (int k = 0; k < 3; k++)
                        q[k] = ((prm.dA[k] * (prm.i0[0] + lo[0] + x)) + prm.dB[k] * (prm.i0[1] + lo[1] + y)) +
                               prm.dC[k] * (prm.i0[2] + lo[2] + 2 * i + h);
                    // The far sums are finite, unless an atom overflows them (a charge of infinity, a tip's
                    // charges beside an atom beyond 1e19 A): all atoms then.
                    bool near_only = listed;
                    float far[8] = {};  // component k of the far sums, from the lines again
                    if (listed) {
#pragma unroll 1
                        for (int k = 0; k < NC; k++) {
                            float v = 0.f;
#pragma unroll 1
                            for (int e = 0; e < N2; e++) {
                                const int y0 = e / N, c0 = e % N;
                                v = fmaf(s_wy[y][y0] * s_wz[h][c0][i],
                                         reinterpret_cast<const float *>(line)[(k * XS + x) * N2 + (c0 >> 1) * 2 * N + 2 * y0 + (c0 & 1)], v);
                            }
                            far[k < NC1 ? k : k - NC1 + 4] = v;
                            near_only = near_only && fabsf(v) <= 3.4e38f;
                        }
                    }
                    if (near_only) {
                        f = box_point_slow<MODE, WITH_E>(prm, df_from(q[0]), df_from(q[1]), df_from(q[2]), s_near, wide, nnear, nch,
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

template <int MODE, bool WITH_E, bool ORTHO, int N>
static int launch_box(const FFParams &prm, BoxPrm B, cudaStream_t st) {
    constexpr int up = (int)BoxUpSmem<MODE, WITH_E, N>::size, leaf = (int)BoxSmem<MODE, WITH_E, N>::size;
    PPGPU_CUDA(cudaFuncSetAttribute(box_up_kernel<MODE, WITH_E, ORTHO, N>, cudaFuncAttributeMaxDynamicSharedMemorySize, up), "ff_box shared memory");
    PPGPU_CUDA(cudaFuncSetAttribute(ff_box_kernel<MODE, WITH_E, ORTHO, N>, cudaFuncAttributeMaxDynamicSharedMemorySize, leaf), "ff_box shared memory");
    for (B.level = B.levels; B.level >= 0; B.level--) {
        long long n = 1;
        for (int k = 0; k < 3; k++) n *= ((B.nb[k] - 1) >> B.level) + 1;
        if (n > 0x0fffffffLL) return set_error(PPGPU_ERR_ARG, "ff grid too large (%lld boxes)", n);
        if (B.level > 0) {
            int rc = launch_box_up(box_up_kernel<MODE, WITH_E, ORTHO, N>, up, n, prm, B, st);
            if (rc) return rc;
        } else {
            ff_box_kernel<MODE, WITH_E, ORTHO, N><<<(unsigned)n, BOX_NT, leaf, st>>>(prm, B);
            PPGPU_CHECK_LAUNCH("ff_box_kernel launch");
        }
    }
    return set_ok();
}

template <int MODE, int N>
static int launch_box_mode(const FFParams &prm, const BoxPrm &B, bool with_e, bool ortho, cudaStream_t st) {
    if (with_e) return ortho ? launch_box<MODE, true, true, N>(prm, B, st) : launch_box<MODE, true, false, N>(prm, B, st);
    return ortho ? launch_box<MODE, false, true, N>(prm, B, st) : launch_box<MODE, false, false, N>(prm, B, st);
}

template <int N>
static int launch_box_nodes(const FFParams &prm, const BoxPrm &B, int mode, bool with_e, bool ortho, cudaStream_t st) {
    switch (mode) {
        case M_LJ:
            return launch_box_mode<M_LJ, N>(prm, B, with_e, ortho, st);
        case M_COUL:
            return launch_box_mode<M_COUL, N>(prm, B, with_e, ortho, st);
        case M_LJC:
            return launch_box_mode<M_LJC, N>(prm, B, with_e, ortho, st);
        default:
            return launch_box_mode<M_QZS, N>(prm, B, with_e, ortho, st);
    }
}

}  // namespace ppgpu
