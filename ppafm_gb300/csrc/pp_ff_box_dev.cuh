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

constexpr int BOX_N = 8;         // nodes per axis
constexpr int BOX_N3 = 512;
constexpr int BOX_S = 16;        // points per axis of a leaf, at most
constexpr int BOX_NT = 256;      // threads of a leaf's CTA
constexpr int BOX_LEVELS = 3;    // levels above the leaves, at most
constexpr int BOX_STAGE = 2 * BOX_NT;   // near atoms staged at a time (the space of a leaf's atom tiles)
constexpr int BOX_NEAR = 2048;          // near atoms listed, as 16-bit indices (half of it as 32-bit ones)
constexpr double BOX_KAPPA = 7.0;

struct BoxPrm {
    int s[3];    // leaf size in points (the last box of an axis may be smaller)
    int nb[3];   // leaves per axis
    int level;   // of this launch: 0 = leaves
    int levels;  // levels above the leaves
    float far2[BOX_LEVELS + 1];   // (7 H)^2, with the tip charges' offsets added to 7 H
    float rep[BOX_LEVELS + 1];    // bound on 12 c12 / (6 c6 r^14), see box_far
    dfl step[3][3];               // rows: grid steps along the axes
    // Offsets of a run's points (every second point of a column) from its middle: a part of few
    // bits, which a displacement's high part takes exactly, and the rest.
    float offh[3][8], offl[3][8];
};

// ---------------------------------------------------------------- interpolation tables

// Chebyshev nodes cos((2k + 1) pi / 16).
struct ChebNodes {
    double t[BOX_N] = {0.98078528040323044913, 0.83146961230254523708, 0.55557023301960222474, 0.19509032201612826785,
                       -0.19509032201612826785, -0.55557023301960222474, -0.83146961230254523708, -0.98078528040323044913};
    double w[BOX_N] = {};  // 1 / prod_{j != k} (t_k - t_j)
    constexpr ChebNodes() {
        for (int k = 0; k < BOX_N; k++) {
            double p = 1.0;
            for (int j = 0; j < BOX_N; j++)
                if (j != k) p *= t[k] - t[j];
            w[k] = 1.0 / p;
        }
    }
};

// Weights [points of the axis][point][node] of evenly spaced points over [-1, 1].
struct ChebPoints {
    float w[BOX_S + 1][BOX_S][BOX_N] = {}, l[BOX_S + 1][BOX_S][BOX_N] = {};  // high and low parts
    constexpr ChebPoints() {
        constexpr ChebNodes c;
        for (int m = 1; m <= BOX_S; m++)
            for (int i = 0; i < m; i++)
                for (int k = 0; k < BOX_N; k++) {
                    const double x = m > 1 ? (2.0 * i - (m - 1)) / (m - 1) : 0.0;
                    double p = c.w[k];
                    for (int j = 0; j < BOX_N; j++)
                        if (j != k) p *= x - c.t[j];
                    w[m][i][k] = (float)p;
                    l[m][i][k] = (float)(p - (double)w[m][i][k]);
                }
    }
};
static __device__ const ChebPoints c_cheb_points = ChebPoints();

// The nodes and their weights as double-floats.
struct ChebNodesDf {
    float th[BOX_N] = {}, tl[BOX_N] = {}, wh[BOX_N] = {}, wl[BOX_N] = {};
    constexpr ChebNodesDf() {
        constexpr ChebNodes c;
        for (int k = 0; k < BOX_N; k++) {
            th[k] = (float)c.t[k];
            tl[k] = (float)(c.t[k] - (double)th[k]);
            wh[k] = (float)c.w[k];
            wl[k] = (float)(c.w[k] - (double)wh[k]);
        }
    }
};
static __constant__ ChebNodesDf c_cheb = ChebNodesDf();
__device__ __forceinline__ dfl cheb_t(int k) { return {c_cheb.th[k], c_cheb.tl[k]}; }

// Lagrange basis polynomial k at x.
__device__ __forceinline__ dfl cheb_basis(int k, dfl x) {
    dfl p = {c_cheb.wh[k], c_cheb.wl[k]};
#pragma unroll 1
    for (int j = 0; j < BOX_N; j++)
        if (j != k) p = df_mul(p, df_add(x, df_neg(cheb_t(j))));
    return p;
}

// -------------------------------------------------------------------------- geometry

// First and last point of box b of an axis at a level.
__device__ __forceinline__ void box_span(const FFParams &prm, const BoxPrm &B, int level, int axis, int b, int &lo, int &hi) {
    lo = (b << level) * B.s[axis];
    hi = min(prm.ns[axis], ((b + 1) << level) * B.s[axis]) - 1;
}

// Half extent in grid steps, exact in float32 (a one-point box gets half a step; its weights are
// those of x = 0).
__device__ __forceinline__ float box_half(int lo, int hi) { return hi > lo ? 0.5f * (float)(hi - lo) : 0.5f; }

__device__ __forceinline__ bool box_there(const BoxPrm &B, int level, const int b[3]) {
    return b[0] <= (B.nb[0] - 1) >> level && b[1] <= (B.nb[1] - 1) >> level && b[2] <= (B.nb[2] - 1) >> level;
}

// What a box is handed from the level above lies in the points of its first leaf, in memory that
// is the box's own until it has read it: first the slots of the interpolated sums, one for each
// level, then each level's list of the atoms that no ancestor sums (their number, -1 for too many,
// then 16-bit indices).  Both ends compute from the sizes alone what there is room for.
struct BoxShare {
    float4 *FE;         // first point
    int m1, m2;         // points of the leaf along y, z
    long long d0, d1;   // points of the grid from one x, y to the next
    int pts, slots, room;  // points; those of the slots; those of one level's list (0: no list)
};
template <int NC>
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
    s.pts = m[0] * m[1] * m[2];
    s.slots = B.levels * (NC * BOX_N3 / 4);
    s.room = prm.natoms <= 65536 && s.pts > s.slots ? (s.pts - s.slots) / B.levels : 0;
    return s;
}
__device__ __forceinline__ float4 *share_cell(const BoxShare &s, int e) {
    const int col = e / s.m2, z = e - col * s.m2, x = col / s.m1, y = col - x * s.m1;
    return s.FE + x * s.d0 + y * s.d1 + z;
}
template <int NC>
__device__ __forceinline__ bool share_has_slot(const BoxShare &s, int level) {
    return s.pts >= (level + 1) * (NC * BOX_N3 / 4);
}
template <int NC>
__device__ __forceinline__ float4 *share_slot(const BoxShare &s, int level, int e) {
    return share_cell(s, level * (NC * BOX_N3 / 4) + e);
}
__device__ __forceinline__ int *share_count(const BoxShare &s, int level) {
    return reinterpret_cast<int *>(share_cell(s, s.slots + level * s.room));
}
__device__ __forceinline__ int share_list_size(const BoxShare &s) { return 8 * s.room - 2; }
__device__ __forceinline__ unsigned short *share_list(const BoxShare &s, int level, int i) {
    const int e = i + 2;  // behind the number
    return reinterpret_cast<unsigned short *>(share_cell(s, s.slots + level * s.room + (e >> 3))) + (e & 7);
}

// Whether an atom (negated coordinates in r0, r1) is far from the box of centre c: explicitly
// rounded operations, because the CTAs of several levels have to agree on it.  rep holds
// 33 (7 H)^8: the interpolation error of the r^-13 force is 5e-6 of the term at 7 H and falls
// with (7 H / r)^8, and 33 is its ratio to the 1.5e-7 allowed of the r^-7 force.
template <int MODE>
__device__ __forceinline__ bool box_far(const float4 &r0, const float4 &r1, const float4 &c, float far2, float rep) {
    const float dx = __fadd_rn(c.x, r0.x), dy = __fadd_rn(c.y, r0.y), dz = __fadd_rn(c.z, r1.x);
    const float r2 = __fmaf_rn(dz, dz, __fmaf_rn(dy, dy, __fmul_rn(dx, dx)));
    if (!(r2 >= far2)) return false;
    if (MODE == M_COUL) return true;
    const float r4 = __fmul_rn(r2, r2), r6 = __fmul_rn(r4, r2);
    return __fmul_rn(fabsf(r1.w), rep) <= __fmul_rn(fabsf(r1.z), __fmul_rn(__fmul_rn(r6, r6), r2));
}

// This CTA's box at a level and its points; boxes are numbered along z first.
__device__ __forceinline__ void box_of_cta(const FFParams &prm, const BoxPrm &B, int level, int b[3], int lo[3], int hi[3]) {
    int r = blockIdx.x;
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

// Weight of node k of this box at node pt & 7 of its child pt >> 3 along an axis (0: no such child).
__device__ __forceinline__ dfl box_child_weight(const FFParams &prm, const BoxPrm &B, int level, int a, int ba, int pt, int k) {
    const int c = 2 * ba + (pt >> 3);
    if (c > (B.nb[a] - 1) >> (level - 1)) return {0.f, 0.f};
    int l, h, pl, ph;
    box_span(prm, B, level - 1, a, c, l, h);
    box_span(prm, B, level, a, ba, pl, ph);
    const dfl x = df_add(df_mul_f(cheb_t(pt & 7), box_half(l, h)), {0.5f * (float)(l + h - pl - ph), 0.f});
    return cheb_basis(k, df_div(x, {box_half(pl, ph), 0.f}));
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
template <int MODE, int NT>
__device__ __forceinline__ bool box_pick(const BoxPrm &B, BoxPick<NT> &S, int level, int nanc, const float4 *T, int nj, int want,
                                         bool ok, int &nmid, int &nzero, int &place) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    int c = 2;
    if (ok && tid < nj) {
        const float4 r0 = T[3 * tid], r1 = T[3 * tid + 1];
        c = box_far<MODE>(r0, r1, S.centre[0], B.far2[level], B.rep[level]) ? 1 : 0;
        for (int m = nanc; m > 0; m--)
            if (box_far<MODE>(r0, r1, S.centre[m], B.far2[level + m], B.rep[level + m])) c = 2;
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

// A tile's atoms of class 0 (n of them, in `left`, after `before` others) to the children's lists, a
// warp for a child.
template <int NC, int NT>
__device__ __forceinline__ void box_leave(const FFParams &prm, const BoxPrm &B, int level, const int b[3], const unsigned short *left,
                                          int n, int before) {
#pragma unroll 1
    for (int q = threadIdx.x >> 5; q < 8; q += NT / 32) {
        const int ch[3] = {2 * b[0] + (q >> 2), 2 * b[1] + ((q >> 1) & 1), 2 * b[2] + (q & 1)};
        if (!box_there(B, level - 1, ch)) continue;
        const BoxShare cs = box_share<NC>(prm, B, level - 1, ch);
        const int m = cs.room > 0 ? min(n, share_list_size(cs) - before) : 0;
        for (int i = threadIdx.x & 31; i < m; i += 32) *share_list(cs, level - 1, before + i) = left[i];
    }
}

// The number of the children's atoms in front of their lists.
template <int NC>
__device__ __forceinline__ void box_leave_count(const FFParams &prm, const BoxPrm &B, int level, const int b[3], int n) {
    const int q = threadIdx.x;
    if (q >= 8) return;
    const int ch[3] = {2 * b[0] + (q >> 2), 2 * b[1] + ((q >> 1) & 1), 2 * b[2] + (q & 1)};
    if (!box_there(B, level - 1, ch)) return;
    const BoxShare cs = box_share<NC>(prm, B, level - 1, ch);
    if (cs.room > 0) *share_count(cs, level - 1) = n <= share_list_size(cs) ? n : -1;
}

// ------------------------------------------------------------------------------ host

// The leaves of a grid and the levels above them; half0: half diagonal of a leaf.  Far at a level:
// kappa half diagonals, and the reach of the tip's charges.
static inline void box_plan(const FFParams &prm, double kappa, double reach, BoxPrm *B, double *half0) {
    memset(B, 0, sizeof(*B));
    for (int k = 0; k < 3; k++) {
        const int parts = (prm.ns[k] + BOX_S - 1) / BOX_S;
        B->s[k] = (prm.ns[k] + parts - 1) / parts;
        if (k == 2) B->s[k] = (B->s[k] + 1) / 2 * 2;  // two threads a column
        B->nb[k] = (prm.ns[k] + B->s[k] - 1) / B->s[k];
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
        double H2 = 0.0;  // half diagonal of a whole box
        for (int c = 0; c < 4; c++) {
            double r2 = 0.0;
            for (int k = 0; k < 3; k++) {
                const double e0 = 0.5 * ((B->s[0] << l) - 1), e1 = 0.5 * ((B->s[1] << l) - 1), e2 = 0.5 * ((B->s[2] << l) - 1);
                const double v = e0 * prm.dA[k] + (c & 1 ? -e1 : e1) * prm.dB[k] + (c & 2 ? -e2 : e2) * prm.dC[k];
                r2 += v * v;
            }
            H2 = std::max(H2, r2);
        }
        const double H = sqrt(H2), R = kappa * H + reach;
        if (l == 0) *half0 = H;
        B->far2[l] = (float)(R * R);
        B->rep[l] = (float)std::min(33.0 * pow(kappa * H, 8.0), 3e38);
    }
}

}  // namespace ppgpu
