// pp_ff_box_dev.cuh -- what the kernels that sum force fields by boxes share (pp_ff_box.cu,
// pp_ff_tip.cu): the boxes' geometry, Chebyshev nodes and weights, the classification of the atoms and
// what a box hands to its children.  pp_ff_box.cu describes the method.
#pragma once

#include <algorithm>
#include <cmath>
#include <cstring>

#include "pp_common.cuh"
#include "pp_df.cuh"
#include "pp_ff_dev.cuh"

namespace ppgpu {

// N, below: nodes per axis, 8 or 10.
constexpr int BOX_S = 16;        // points per axis of a leaf, at most
constexpr int BOX_NT = 256;      // threads of a leaf's CTA
constexpr int BOX_LEVELS = 3;    // levels above the leaves, at most
constexpr int BOX_STAGE = BOX_NT;       // near atoms staged at a time
constexpr int BOX_LEFT = 4096;          // atoms that a CTA of an upper box leaves to the children
constexpr int BOX_NEAR = 1024;          // near atoms listed, as 16-bit indices (half of it as 32-bit ones)

// Indices of a leaf's near atoms, in either width (wide: more than 65536 atoms).
union BoxNear {
    unsigned short h[BOX_NEAR];
    int w[BOX_NEAR / 2];
    __device__ __forceinline__ int at(bool wide, int i) const { return wide ? w[i] : (int)h[i]; }
    __device__ __forceinline__ void set(bool wide, int i, int j) {
        if (wide) w[i] = j;
        else h[i] = (unsigned short)j;
    }
};
static_assert(alignof(BoxNear) == alignof(int), "32-bit access");

struct BoxPrm {
    int s[3];    // points of a leaf along an axis, one more for the first rem[axis] leaves; the last may have fewer
    int rem[3];
    int nb[3];   // leaves per axis
    int level;   // of this launch: 0 = leaves
    int levels;  // levels above the leaves
    float far2[BOX_LEVELS + 1];   // (kappa H)^2, with the tip charges' offsets added to kappa H
    float rep[BOX_LEVELS + 1];    // bound on 12 c12 / (6 c6 r^14), see box_far
    dfl step[3][3];               // rows: grid steps along the axes
    // Offsets of a run's points (every second point of a column) from its middle: a part of few
    // bits, which a displacement's high part takes exactly, and the rest.
    float offh[3][8], offl[3][8];
};

// ---------------------------------------------------------------- interpolation tables

// Chebyshev nodes cos((2k + 1) pi / 2N).
template <int N>
struct ChebNodes {
    double t[N] = {}, w[N] = {};  // w: 1 / prod_{j != k} (t_k - t_j)
    constexpr ChebNodes() {
        constexpr double t8[4] = {0.98078528040323044913, 0.83146961230254523708, 0.55557023301960222474, 0.19509032201612826785};
        constexpr double t10[5] = {0.98768834059513772619, 0.89100652418836786236, 0.70710678118654752440, 0.45399049973954679156,
                                   0.15643446504023086901};
        static_assert(N == 8 || N == 10, "nodes");
        for (int k = 0; k < N / 2; k++) {
            t[k] = N == 8 ? t8[k < 4 ? k : 3] : t10[k];
            t[N - 1 - k] = -t[k];
        }
        for (int k = 0; k < N; k++) {
            double p = 1.0;
            for (int j = 0; j < N; j++)
                if (j != k) p *= t[k] - t[j];
            w[k] = 1.0 / p;
        }
    }
};

// Weights [points of the axis][point][node] of evenly spaced points over [-1, 1]; LOW: what float32
// leaves of them.
template <int N, bool LOW>
struct ChebPoints {
    float w[BOX_S + 1][BOX_S][N] = {};
    constexpr ChebPoints() {
        constexpr ChebNodes<N> c;
        for (int m = 1; m <= BOX_S; m++)
            for (int i = 0; i < m; i++)
                for (int k = 0; k < N; k++) {
                    const double x = m > 1 ? (2.0 * i - (m - 1)) / (m - 1) : 0.0;
                    double p = c.w[k];
                    for (int j = 0; j < N; j++)
                        if (j != k) p *= x - c.t[j];
                    w[m][i][k] = LOW ? (float)(p - (double)(float)p) : (float)p;
                }
    }
};
static __device__ const ChebPoints<8, false> c_points8 = ChebPoints<8, false>();
static __device__ const ChebPoints<10, false> c_points10 = ChebPoints<10, false>();
template <int N>
__device__ __forceinline__ const ChebPoints<N, false> &cheb_points() {
    if constexpr (N == 8) return c_points8;
    else return c_points10;
}

// The nodes and their weights as double-floats.
template <int N>
struct ChebNodesDf {
    float th[N] = {}, tl[N] = {}, wh[N] = {}, wl[N] = {};
    constexpr ChebNodesDf() {
        constexpr ChebNodes<N> c;
        for (int k = 0; k < N; k++) {
            th[k] = (float)c.t[k];
            tl[k] = (float)(c.t[k] - (double)th[k]);
            wh[k] = (float)c.w[k];
            wl[k] = (float)(c.w[k] - (double)wh[k]);
        }
    }
};
static __constant__ ChebNodesDf<8> c_nodes8 = ChebNodesDf<8>();
static __constant__ ChebNodesDf<10> c_nodes10 = ChebNodesDf<10>();
template <int N>
__device__ __forceinline__ const ChebNodesDf<N> &cheb_nodes() {
    if constexpr (N == 8) return c_nodes8;
    else return c_nodes10;
}
template <int N>
__device__ __forceinline__ dfl cheb_t(int k) {
    return {cheb_nodes<N>().th[k], cheb_nodes<N>().tl[k]};
}

// The Lagrange basis polynomials at x, from the products of the factors before and behind each.
template <int N, class Store>
__device__ __forceinline__ void cheb_row(dfl x, Store store) {
    dfl behind[N];
    dfl p = {1.f, 0.f};
#pragma unroll
    for (int k = N - 1; k >= 0; k--) {
        behind[k] = p;
        p = df_mul(p, df_add(x, df_neg(cheb_t<N>(k))));
    }
    p = {1.f, 0.f};
#pragma unroll
    for (int k = 0; k < N; k++) {
        store(k, df_mul(df_mul(p, behind[k]), {cheb_nodes<N>().wh[k], cheb_nodes<N>().wl[k]}));
        p = df_mul(p, df_add(x, df_neg(cheb_t<N>(k))));
    }
}

// -------------------------------------------------------------------------- geometry

// First and last point of box b of an axis at a level.
__device__ __forceinline__ void box_span(const FFParams &prm, const BoxPrm &B, int level, int axis, int b, int &lo, int &hi) {
    const int first = b << level, end = (b + 1) << level;
    lo = first * B.s[axis] + min(first, B.rem[axis]);
    hi = min(prm.ns[axis], end * B.s[axis] + min(end, B.rem[axis])) - 1;
}

// Half extent in grid steps, exact in float32 (a one-point box gets half a step; its weights are
// those of x = 0).
__device__ __forceinline__ float box_half(int lo, int hi) { return hi > lo ? 0.5f * (float)(hi - lo) : 0.5f; }

__device__ __forceinline__ bool box_there(const BoxPrm &B, int level, const int b[3]) {
    return b[0] <= (B.nb[0] - 1) >> level && b[1] <= (B.nb[1] - 1) >> level && b[2] <= (B.nb[2] - 1) >> level;
}

// What a box is handed from the level above lies in the points of its first leaf, in memory that
// is the box's own until it has read it: the interpolated sums, then the list of the atoms that no
// ancestor sums (their number, -1 for too many, then 16-bit indices).  The box leaves the same to
// its children, to the first one in the same place: it has read its sums by then, and the list
// it writes runs behind the tiles that it has read.  Both ends compute from the sizes alone what
// there is room for.
struct BoxShare {
    float4 *FE;         // first point
    int m1, m2;         // points of the leaf along y, z
    long long d0, d1;   // points of the grid from one x, y to the next
    int pts, room;      // points; those for the list (0: no list)
    float r1, r2;       // 1 / m1, 1 / m2
};
template <int N, int NC>
__device__ __forceinline__ BoxShare box_share(const FFParams &prm, const BoxPrm &B, int level, const int b[3]) {
    int lo[3], m[3];
#pragma unroll
    for (int k = 0; k < 3; k++) {
        int hi;
        box_span(prm, B, 0, k, b[k] << level, lo[k], hi);
        m[k] = hi - lo[k] + 1;
    }
    BoxShare s;
    s.d1 = prm.ns[2];
    s.d0 = (long long)prm.ns[1] * prm.ns[2];
    s.FE = prm.FE + lo[0] * s.d0 + lo[1] * s.d1 + lo[2];
    s.m1 = m[1];
    s.m2 = m[2];
    s.r1 = __fdiv_rn(1.f, (float)m[1]);
    s.r2 = __fdiv_rn(1.f, (float)m[2]);
    s.pts = m[0] * m[1] * m[2];
    s.room = prm.natoms <= 65536 ? max(0, s.pts - NC * (N * N * N / 4)) : 0;
    return s;
}
__device__ __forceinline__ float4 *share_cell(const BoxShare &s, int e) {
    // quotients of numbers up to 4096 by 16 at most: the rounding stays far below the half added
    const int col = (int)(((float)e + 0.5f) * s.r2), z = e - col * s.m2;
    const int x = (int)(((float)col + 0.5f) * s.r1), y = col - x * s.m1;
    return s.FE + x * s.d0 + y * s.d1 + z;
}
// Whether there is room for the sums: cells 0 to NC N^3 / 4 - 1, NC components of the nodes.
template <int N, int NC>
__device__ __forceinline__ bool share_has_sums(const BoxShare &s) {
    return s.pts >= NC * (N * N * N / 4);
}
template <int N, int NC>
__device__ __forceinline__ int *share_count(const BoxShare &s) {
    return reinterpret_cast<int *>(share_cell(s, NC * (N * N * N / 4)));
}
__device__ __forceinline__ int share_list_size(const BoxShare &s) { return 8 * s.room - 2; }
template <int N, int NC>
__device__ __forceinline__ unsigned short *share_list(const BoxShare &s, int i) {
    const int e = i + 2;  // behind the number
    return reinterpret_cast<unsigned short *>(share_cell(s, NC * (N * N * N / 4) + (e >> 3))) + (e & 7);
}

// Whether an atom (negated coordinates in r0, r1) is far from the box of centre c: explicitly
// rounded operations, because the CTAs of several levels have to agree on it.  rep: the interpolation
// error of the r^-13 force at kappa H (5e-6 of the term with 8 nodes at 7, 2e-5 with 10 at 4.25) over
// the 1.5e-7 allowed of the r^-7 force, times (kappa H)^N, with whose power over r it falls.
//   No distance would be enough for an atom without attraction.  Where the r^-13 force is the larger
// one, the error is held against it instead, beyond 1.55 (8 nodes) or 1.63 (10) kappa H.  18540 atoms with c6 = 0 on 200^3
// points: 82 ms with all of them near, 7.2 now, 53 pair by pair; error against 64 bits 2.5e-7, 3.8e-7, 4.1e-7.
template <int MODE, int N>
__device__ __forceinline__ bool box_far(const float4 &r0, const float4 &r1, const float4 &c, float far2, float rep) {
    const float dx = __fadd_rn(c.x, r0.x), dy = __fadd_rn(c.y, r0.y), dz = __fadd_rn(c.z, r1.x);
    const float r2 = __fmaf_rn(dz, dz, __fmaf_rn(dy, dy, __fmul_rn(dx, dx)));
    if (!(r2 >= far2)) return false;
    if (MODE == M_COUL) return true;
    const float c6 = fabsf(r1.z), c12 = fabsf(r1.w);
    const float r4 = __fmul_rn(r2, r2), r8 = __fmul_rn(r4, r4), r6 = __fmul_rn(r4, r2);
    const float rn = N == 8 ? __fmul_rn(r8, r6) : __fmul_rn(r8, r8);  // r^(6 + N)
    if (__fmul_rn(c12, rep) <= __fmul_rn(c6, fminf(rn, 3e38f))) return true;
    const float rN = N == 8 ? r8 : __fmul_rn(r8, r2);
    return rN >= rep && __fmul_rn(c6, r6) <= c12 && c12 <= 3e38f;
}

// A CTA's box at a level and its points; boxes are numbered along z first.
__device__ __forceinline__ void box_of_cta(const FFParams &prm, const BoxPrm &B, int level, int box, int b[3], int lo[3], int hi[3]) {
    int r = box;
    const int n2 = ((B.nb[2] - 1) >> level) + 1, n1 = ((B.nb[1] - 1) >> level) + 1;
    b[2] = r % n2;
    r /= n2;
    b[1] = r % n1;
    b[0] = r / n1;
#pragma unroll
    for (int k = 0; k < 3; k++) box_span(prm, B, level, k, b[k], lo[k], hi[k]);
}

// Centre of this box's ancestor `up` levels above it (0: its own).
__device__ __forceinline__ float4 box_centre(const FFParams &prm, const BoxPrm &B, int level, const int b[3], int up) {
    dfl s[3] = {{0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}};
#pragma unroll
    for (int a = 0; a < 3; a++) {
        int l, h;
        box_span(prm, B, level + up, a, b[a] >> up, l, h);
        const float g = 0.5f * (float)(l + h) + (float)prm.i0[a];
#pragma unroll
        for (int k = 0; k < 3; k++) s[k] = df_add(s[k], df_mul_f(B.step[a][k], g));
    }
    return make_float4(df_round(s[0]), df_round(s[1]), df_round(s[2]), 0.f);
}

// Node i of child c (0 or 1) along an axis, in the box's own [-1, 1]; false: no such child.
template <int N>
__device__ __forceinline__ bool box_child_node(const FFParams &prm, const BoxPrm &B, int level, int a, int ba, int c, int i, dfl &x) {
    if (2 * ba + c > (B.nb[a] - 1) >> (level - 1)) return false;
    int l, h, pl, ph;
    box_span(prm, B, level - 1, a, 2 * ba + c, l, h);
    box_span(prm, B, level, a, ba, pl, ph);
    x = df_div(df_add(df_mul_f(cheb_t<N>(i), box_half(l, h)), {0.5f * (float)(l + h - pl - ph), 0.f}), {box_half(pl, ph), 0.f});
    return true;
}

// What the threads of a CTA share while they go through the atoms.
template <int NT>
struct BoxPick {
    int cnt[2][NT / 32];
    float4 centre[BOX_LEVELS + 1];  // this box's (0) and its ancestors'
    unsigned char mid[NT];          // atoms of the wanted class in the tile
};

// Classifies the atoms of tile T, one a thread.  0: near (leaves sum them at the points, upper boxes
// leave them to their children), 1: far, on this machine's nodes, 2: an ancestor's.  Lists those of
// class `want` in S.mid (nmid of them); nzero: number of class 0; place: where this thread's atom
// comes among those (-1: not one).  Threads must meet before they read S.mid.  False when a
// thread's tile did not land.
template <int MODE, int N, int NT>
__device__ __forceinline__ bool box_pick(const BoxPrm &B, BoxPick<NT> &S, int level, int nanc, const float4 *T, int nj, int want,
                                         bool ok, int &nmid, int &nzero, int &place) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    int c = 2;
    if (ok && tid < nj) {
        const float4 r0 = T[3 * tid], r1 = T[3 * tid + 1];
        c = box_far<MODE, N>(r0, r1, S.centre[0], B.far2[level], B.rep[level]) ? 1 : 0;
        for (int m = nanc; m > 0; m--)
            if (box_far<MODE, N>(r0, r1, S.centre[m], B.far2[level + m], B.rep[level + m])) c = 2;
    }
    const unsigned bm = __ballot_sync(0xffffffffu, c == want), bz = __ballot_sync(0xffffffffu, c == 0);
    if (lane == 0) {
        S.cnt[0][warp] = __popc(bm);
        S.cnt[1][warp] = __popc(bz);
    }
    if (__syncthreads_or(!ok)) return false;
    const unsigned lt = (1u << lane) - 1u;
    nmid = nzero = 0;
    int m0 = 0, z0 = 0;
#pragma unroll
    for (int g = 0; g < NT / 32; g++) {
        if (g == warp) {
            m0 = nmid;
            z0 = nzero;
        }
        nmid += S.cnt[0][g];
        nzero += S.cnt[1][g];
    }
    if (c == want) S.mid[m0 + __popc(bm & lt)] = (unsigned char)tid;
    place = c == 0 ? z0 + __popc(bz & lt) : -1;
    return true;
}

// Record j into place tid of a tile; .w of its last part: charged.
__device__ __forceinline__ void box_gather(const FFParams &prm, float4 *T, int j) {
    const float4 *a = prm.atoms + (size_t)j * FF_REC;
    const float4 c = ldg4(a + 2);
    T[0] = ldg4(a);
    T[1] = ldg4(a + 1);
    T[2] = make_float4(c.x, c.y, c.z, j < prm.ncharged ? 1.f : 0.f);
}

// The atoms that this CTA leaves to the children of its box (n of them, in `left`; none of them
// when there are more), behind `before` others of `all`: their lists, and from one CTA the number.
template <int N, int NC, int NT>
__device__ __forceinline__ void box_leave(const FFParams &prm, const BoxPrm &B, int level, const int b[3], const unsigned short *left,
                                          int n, int before, int all, bool number) {
    if (all < 0) n = 0;
#pragma unroll 1
    for (int q = threadIdx.x >> 5; q < 8; q += NT / 32) {
        const int ch[3] = {2 * b[0] + (q >> 2), 2 * b[1] + ((q >> 1) & 1), 2 * b[2] + (q & 1)};
        if (!box_there(B, level - 1, ch)) continue;
        const BoxShare cs = box_share<N, NC>(prm, B, level - 1, ch);
        if (cs.room == 0) continue;
        const int m = min(n, share_list_size(cs) - before), lane = threadIdx.x & 31;
        for (int i = lane; i < m; i += 32) *share_list<N, NC>(cs, before + i) = left[i];
        if (number && lane == 0) *share_count<N, NC>(cs) = all <= share_list_size(cs) ? all : -1;
    }
}

// ----------------------------------------------------------------------- clusters
//
// An upper box may be worked on by the CTAs of a cluster: each takes a part of the atoms and some
// of the children, and reads the others' sums of the nodes from their shared memory.

__device__ __forceinline__ int cluster_rank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return (int)r;
}
__device__ __forceinline__ int cluster_size() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
    return (int)r;
}
__device__ __forceinline__ void cluster_meet() {
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ uint32_t cluster_addr(const void *p, int rank) {
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
    return a;
}
__device__ __forceinline__ float4 cluster_ld4(uint32_t a) {
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ int cluster_ldi(uint32_t a) {
    int v;
    asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ void async_copy16(void *dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// ------------------------------------------------------------------------------ host

// Leaves of a grid.
static inline double box_count(const FFParams &prm) {
    double n = 1.0;
    for (int k = 0; k < 3; k++) n *= (prm.ns[k] + BOX_S - 1) / BOX_S;
    return n;
}

// The leaves of a grid and the levels above them; half0: H of a leaf.  Far at a level: kappa H, and
// the reach of the tip's charges.  H is the half diagonal, or that of a cube of the longest
// edge: the error follows the nearest singularity beside the longest edge, and kappa is a cube's.
static inline void box_plan(const FFParams &prm, int N, double kappa, double reach, BoxPrm *B, double *half0) {
    memset(B, 0, sizeof(*B));
    for (int k = 0; k < 3; k++) {
        B->nb[k] = (prm.ns[k] + BOX_S - 1) / BOX_S;
        if (B->nb[k] == 0) continue;  // no points
        B->s[k] = (prm.ns[k] + B->nb[k] - 1) / B->nb[k];
        if (k == 2) B->s[k] = (B->s[k] + 1) / 2 * 2;  // two threads a column
        // Whole leaves and a smaller last one, unless that is too small to be handed sums.
        if (prm.ns[k] - (B->nb[k] - 1) * B->s[k] < (N == 8 ? 8 : 12)) {
            B->s[k] = prm.ns[k] / B->nb[k];
            B->rem[k] = prm.ns[k] % B->nb[k];
        }
    }
    const double *d[3] = {prm.dA, prm.dB, prm.dC};
    for (int a = 0; a < 3; a++)
        for (int k = 0; k < 3; k++) B->step[a][k] = df_from(d[a][k]);
    for (int k = 0; k < 3; k++)
        for (int i = 0; i < 8; i++) {
            const double v = prm.dC[k] * (2 * i - 7);
            const double h = rint(v * 8192.0) / 8192.0;  // multiples of 2^-13
            B->offh[k][i] = (float)h;
            B->offl[k][i] = (float)(v - (double)(float)h);
        }
    for (int l = 0; l <= BOX_LEVELS; l++) {
        double e[3], H2 = 0.0;  // half extents of the largest box, in steps
        for (int k = 0; k < 3; k++) e[k] = 0.5 * ((B->s[k] << l) + std::min(1 << l, B->rem[k]) - 1);
        for (int c = 0; c < 4; c++) {
            double r2 = 0.0;
            for (int k = 0; k < 3; k++) {
                const double v = e[0] * prm.dA[k] + (c & 1 ? -e[1] : e[1]) * prm.dB[k] + (c & 2 ? -e[2] : e[2]) * prm.dC[k];
                r2 += v * v;
            }
            H2 = std::max(H2, r2);
        }
        for (int a = 0; a < 3; a++) {
            double r2 = 0.0;
            for (int k = 0; k < 3; k++) r2 += e[a] * d[a][k] * e[a] * d[a][k];
            H2 = std::max(H2, 3.0 * r2);
        }
        const double H = sqrt(H2), R = kappa * H + reach;
        if (l == 0) *half0 = H;
        B->far2[l] = (float)(R * R);
        B->rep[l] = (float)std::min((N == 8 ? 33.0 : 130.0) * pow(kappa * H, (double)N), 3e38);
    }
}

// Points of a leaf (a smaller one where their sizes differ).
static inline int box_leaf(const BoxPrm &B) { return B.s[0] * B.s[1] * B.s[2]; }

// CTAs of a cluster for each of n upper boxes: enough to fill the SMs (two CTAs each).
static inline int box_cluster(long long n) {
    int c = 1;
    while (c < 8 && n * c < 456) c *= 2;
    return c;
}

// A level above the leaves: n boxes, a cluster of CTAs each.
template <class Kernel>
static int launch_box_up(Kernel kernel, int smem, long long n, const FFParams &prm, const BoxPrm &B, cudaStream_t st) {
    const int c = box_cluster(n);
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)c;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3((unsigned)(n * c));
    cfg.blockDim = dim3(BOX_NT);
    cfg.dynamicSmemBytes = (size_t)smem;
    cfg.stream = st;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    PPGPU_CUDA(cudaLaunchKernelEx(&cfg, kernel, prm, B), "ff box launch");
    return PPGPU_OK;
}

int launch_ff_box10(const FFParams &prm, const BoxPrm &B, int mode, bool with_e, bool ortho, cudaStream_t st);  // pp_ff_box10.cu

}  // namespace ppgpu
