// pp_ff_tip.cu -- the pz and dz2 Coulomb tips in double-float, directly and by boxes.
//
// getCoulombFF's finite-difference tips (ppafm/cpp/ProbeParticle.cpp:192-209): the Coulomb field of
// the same charge at heights dz - h, dz and dz + h (h = 0.1 A) with weights (-1, 0, 1)/h for pz and
// (1, -2, 1)/h^2 for dz2.  The differences cancel (r/h)^2 of the significand, so they are formed
// in double-float (pp_df.cuh, ~46 bits after the reciprocal root), as are the sums over the
// atoms: what is left is the rounding of the stored float32, as in float64.  Float64 itself
// issues at 1/64 of the float32 rate here, which made these tips 400 times an s tip.
//
// Bound by float32 instructions (~210 a pair for dz2, no memory traffic to speak of).
//   342 charges on 200^3 points: dz2 423 ms in float64, 16.7 ms pair by pair here, 1.86 by boxes (error
//   against 64 bits 5.6e-8 in all three: the stored float32's rounding).
#include "pp_ff_box_dev.cuh"

namespace ppgpu {

// A thread's run of positions along one column: the in-plane distance of an atom is formed once
// for all of them, and the sums (6 to 10 registers each) fit 128 registers (runs of 6 and 8 spill).
constexpr int TIP_P = 4;
constexpr int TIP_THREADS = 128;
constexpr double TIP_H = 0.1;

// acc += t; the low part collects the errors and is folded in at the end of an atom tile.
__device__ __forceinline__ void df_acc(dfl &acc, dfl t) {
    const dfl s = two_sum(acc.h, t.h);
    acc.h = s.h;
    acc.l = __fadd_rn(acc.l, __fadd_rn(s.l, t.l));
}

// 1/r and 1/r^3 of r^2: the approximate root y, then the series of (1 - e)^(-1/2) in its exact
// residual e = 1 - r^2 y^2 (|e| < 2^-20, so two terms).
struct InvR {
    dfl i1, i3;
};
__device__ __forceinline__ InvR inv_r(dfl r2) {
    const float y = rsqrt_approx(r2.h);
    const dfl y2 = two_prod(y, y);
    const dfl p = two_prod(r2.h, y2.h);
    float e = __fsub_rn(__fsub_rn(1.f, p.h), p.l);
    e = __fmaf_rn(-r2.h, y2.l, e);
    e = __fmaf_rn(-r2.l, y2.h, e);
    const float d = __fmul_rn(e, __fmaf_rn(0.375f, e, 0.5f));  // 1/r = y (1 + d)
    const dfl y3 = two_prod(y, y2.h);
    InvR o;
    o.i1 = {y, __fmul_rn(y, d)};
    // (1 + d)^3 = 1 + 3 d (1 + d) + d^3, the cube below 2^-60
    o.i3 = {y3.h, __fmaf_rn(y3.h, __fmul_rn(3.f, __fmaf_rn(d, d, d)), __fmaf_rn(y, y2.l, y3.l))};
    return o;
}

// Sums of TIP_P positions: force, the axial part of the z force before its factor h, energy; without
// the tip's weight (1/h or 1/h^2).
struct TipSums {
    dfl F[3][TIP_P], A[TIP_P], E[TIP_P];
    __device__ __forceinline__ void zero() {
#pragma unroll
        for (int i = 0; i < TIP_P; i++) F[0][i] = F[1][i] = F[2][i] = A[i] = E[i] = {0.f, 0.f};
    }
    // Folds the collected low parts in.
    template <bool WITH_E>
    __device__ __forceinline__ void fold() {
#pragma unroll
        for (int i = 0; i < TIP_P; i++) {
#pragma unroll
            for (int k = 0; k < 3; k++) F[k][i] = two_sum(F[k][i].h, F[k][i].l);
            A[i] = two_sum(A[i].h, A[i].l);
            if (WITH_E) E[i] = two_sum(E[i].h, E[i].l);
        }
    }
    // Component k (x, y, z, energy) of position i.
    __device__ __forceinline__ dfl get(int k, int i) const {
        if (k == 2) return df_add(F[2][i], df_mul_raw(A[i], df_from(TIP_H)));
        return k == 3 ? E[i] : F[k][i];
    }
};

// A part of an atom record (k: 0 x, y; 1 z; 2 charge) with finite coordinates (and their low parts) of
// 1e18 A at most: from there on a charge's field is nothing in float32, and r^2 would overflow.
__device__ __forceinline__ float4 tip_record(float4 v, int k) {
    auto lim = [](float &h, float &l) {
        if (!(fabsf(h) > 1e18f && fabsf(h) <= 3.4e38f)) return;
        h = copysignf(1e18f, h);
        l = 0.f;
    };
    if (k == 0) {
        lim(v.x, v.z);
        lim(v.y, v.w);
    } else if (k == 1) {
        lim(v.x, v.y);
    }
    return v;
}
__device__ __forceinline__ void tip_limit(float4 *record) {
    record[0] = tip_record(record[0], 0);
    record[1] = tip_record(record[1], 1);
}

// Adds a charge q (negated coordinates in r0, r1) to the sums at positions p (x and y of the first
// one only when ORTHO).
template <int KIND, bool WITH_E, bool ORTHO>
__device__ __forceinline__ void tip_add(const dfl (*p)[TIP_P], const float4 &r0, const float4 &r1, float q, TipSums &S) {
    const dfl h2 = df_from(2 * TIP_H), hh = df_from(TIP_H * TIP_H), eps = df_from(1.0e-8);
    dfl dx, dy, s, shh;
#pragma unroll
    for (int i = 0; i < TIP_P; i++) {
        if (i == 0 || !ORTHO) {
            dx = df_add(p[0][i], {r0.x, r0.z});
            dy = df_add(p[1][i], {r0.y, r0.w});
            s = df_add(df_add(df_sq(dx), df_sq(dy)), eps);
            shh = df_add(s, hh);
        }
        const dfl dz = df_add(p[2][i], {r1.x, r1.y}), zz = df_sq(dz);
        const dfl a = df_add(shh, zz), b = df_mul_raw(dz, h2);  // r^2 + h^2, 2 h dz
        const InvR up = inv_r(df_add(a, b)), dn = inv_r(df_add(a, df_neg(b)));
        const dfl D = df_add_raw(up.i3, df_neg(dn.i3)), T = df_add_raw(up.i3, dn.i3);
        dfl rad, e;  // the field is q (rad (dx, dy, dz) + h ax z), ax = T (pz) or D (dz2)
        if (KIND == 1) {
            rad = D;
            if (WITH_E) e = df_add_raw(up.i1, df_neg(dn.i1));
        } else {
            const InvR md = inv_r(df_add(s, zz));
            rad = df_add_raw(T, {-2.f * md.i3.h, -2.f * md.i3.l});
            if (WITH_E) e = df_add_raw(df_add_raw(up.i1, dn.i1), {-2.f * md.i1.h, -2.f * md.i1.l});
        }
        rad = df_mul_raw(rad, q);
        df_acc(S.F[0][i], df_mul_raw(rad, dx));
        df_acc(S.F[1][i], df_mul_raw(rad, dy));
        df_acc(S.F[2][i], df_mul_raw(rad, dz));
        df_acc(S.A[i], df_mul_raw(KIND == 1 ? T : D, q));
        if (WITH_E) df_acc(S.E[i], df_mul_raw(e, q));
    }
}

// The sums of position i as the stored value, added to what is there when accumulating.
template <int KIND, bool WITH_E>
__device__ __forceinline__ void tip_store(const FFParams &prm, const TipSums &S, int i, float4 *dst) {
    const float w = KIND == 1 ? 10.f : 100.f;
    float4 o;
    o.x = df_round(df_mul_raw(S.get(0, i), w));
    o.y = df_round(df_mul_raw(S.get(1, i), w));
    o.z = df_round(df_mul_raw(S.get(2, i), w));
    o.w = WITH_E ? df_round(df_mul_raw(S.get(3, i), w)) : 0.f;
    if (prm.accumulate) {
        const float4 old = *dst;
        o = make_float4(o.x + old.x, o.y + old.y, o.z + old.z, o.w + old.w);
    }
    *dst = o;
}

// --------------------------------------------------------------------- pair by pair

template <int KIND, bool WITH_E, bool ORTHO>
__global__ void __launch_bounds__(TIP_THREADS, 4) ff_tip_kernel(const FFParams prm) {
    static_assert(KIND == 1 || KIND == 2, "pz or dz2");
    __shared__ __align__(16) float4 s_at[FF_TILE * FF_REC];
    const int tid = threadIdx.x;
    const long long chunk = (long long)blockIdx.x * TIP_THREADS + tid;
    const bool valid = chunk < prm.nchunks;
    int la = 0, lb = 0, lz0 = 0;
    if (valid) {
        const long long col = chunk / prm.nzc;
        lz0 = (int)(chunk - col * prm.nzc) * TIP_P;
        la = (int)(col / prm.ns[1]);
        lb = (int)(col - (long long)la * prm.ns[1]);
    }
    const double ga = prm.i0[0] + la, gb = prm.i0[1] + lb, gc = prm.i0[2] + lz0;
    dfl p[3][TIP_P];
#pragma unroll
    for (int i = 0; i < TIP_P; i++)
#pragma unroll
        for (int k = 0; k < 3; k++)
            if (k == 2 || i == 0 || !ORTHO) p[k][i] = df_from(((prm.dA[k] * ga) + prm.dB[k] * gb) + prm.dC[k] * (gc + i));
    TipSums S;
    S.zero();
    for (int base = 0; base < prm.ncharged; base += FF_TILE) {
        const int nj = min(FF_TILE, prm.ncharged - base);
        __syncthreads();
        for (int i = tid; i < nj * FF_REC; i += TIP_THREADS) s_at[i] = tip_record(prm.atoms[(size_t)base * FF_REC + i], i % FF_REC);
        __syncthreads();
        for (int j = 0; j < nj; j++) tip_add<KIND, WITH_E, ORTHO>(p, s_at[3 * j], s_at[3 * j + 1], s_at[3 * j + 2].z, S);
        S.fold<WITH_E>();
    }
    if (!valid) return;
    float4 *out = prm.FE + ((long long)la * prm.ns[1] + lb) * prm.ns[2] + lz0;
#pragma unroll
    for (int i = 0; i < TIP_P; i++) {
        if (lz0 + i >= prm.ns[2]) break;
        tip_store<KIND, WITH_E>(prm, S, i, out + i);
    }
}

// ------------------------------------------------------------------------- by boxes
//
// The method of pp_ff_box.cu in double-float: the charges far from a box of up to 16^3 points
// (R >= 5 H + h) are summed on 10^3 nodes, which with the smoother Coulomb terms leaves 4e-10 of a
// pair's field, a hundredth of the stored value's rounding; nodes, weights and sums are
// double-floats.  256 threads: 250 with four of the nodes each; for the points runs of every fourth
// point of a column (neighbours write neighbouring points).  The interpolation goes along x (line),
// then along y for four of the box's x at a time (plane), then along z into a run's sums.  128
// registers, two CTAs a SM.

constexpr double TIP_KAPPA = 5.0;
constexpr int TIP_NT = 256;
constexpr int TIP_N = 10, TIP_N2 = 100, TIP_N3 = 1000;  // nodes
constexpr int TIP_X = 4;  // of the box's x in the plane
static __device__ const ChebPoints<TIP_N, true> c_points_low = ChebPoints<TIP_N, true>();

// acc += w v (both double-floats).
__device__ __forceinline__ void df_fma(dfl &acc, dfl w, dfl v) { df_acc(acc, df_mul_raw(w, v)); }

// Parts of the nodes' positions along the axes.
__device__ __forceinline__ void tip_node_table(const FFParams &prm, const BoxPrm &B, int level, const int b[3], int i, dfl (*node)[TIP_N][3]) {
    const int a = i / TIP_N, n = i % TIP_N;
    int l, h;
    box_span(prm, B, level, a, a == 0 ? b[0] : (a == 1 ? b[1] : b[2]), l, h);
    const dfl g = df_add(df_mul_f(cheb_t<TIP_N>(n), box_half(l, h)), {0.5f * (float)(l + h) + (float)prm.i0[a], 0.f});
#pragma unroll
    for (int k = 0; k < 3; k++) node[a][n][k] = df_mul(B.step[a][k], g);
}

// Positions of a thread's four nodes.
__device__ __forceinline__ void tip_nodes(const dfl (*node)[TIP_N][3], int tid, dfl (*p)[TIP_P]) {
#pragma unroll
    for (int i = 0; i < TIP_P; i++) {
        const int e = min(TIP_P * tid + i, TIP_N3 - 1), ia = e / TIP_N2, ib = e / TIP_N % TIP_N, ic = e % TIP_N;
#pragma unroll
        for (int k = 0; k < 3; k++) p[k][i] = df_add(df_add(node[0][ia][k], node[1][ib][k]), node[2][ic][k]);
    }
}

// Upper boxes, as box_up_kernel: a cluster of CTAs a box, parts of the charges and of the children each.
// Shared memory: an atom tile, then the sums along z; this CTA's sums, then those along y; the
// box's sums.
template <bool WITH_E>
struct TipUpSmem {
    static constexpr int K = WITH_E ? 4 : 3;
    static constexpr size_t own = sizeof(dfl) * K * TIP_N3, sum = 2 * own, size = 3 * own;
    static_assert(own >= sizeof(float4) * TIP_NT * FF_REC, "the tile's space");
};

template <int KIND, bool WITH_E>
__global__ void __launch_bounds__(TIP_NT, 2) tip_up_kernel(const __grid_constant__ FFParams prm, const __grid_constant__ BoxPrm B) {
    using Smem = TipUpSmem<WITH_E>;
    constexpr int K = Smem::K, NC = 2 * K, NT = TIP_NT, C4 = K * TIP_N3 / 2;
    extern __shared__ __align__(128) unsigned char tip_raw[];
    float4 *tile = reinterpret_cast<float4 *>(tip_raw);
    dfl *lz = reinterpret_cast<dfl *>(tip_raw), *own = reinterpret_cast<dfl *>(tip_raw + Smem::own), *sum = reinterpret_cast<dfl *>(tip_raw + Smem::sum);
    __shared__ unsigned short s_left[BOX_LEFT];
    __shared__ int s_count;
    __shared__ BoxPick<NT> pk;
    __shared__ dfl s_node[3][TIP_N][3], s_w[3][2][TIP_N][TIP_N];  // weights: [axis][child][node of the box][node of the child]

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int level = B.level, rank = cluster_rank(), ncta = cluster_size(), nat = prm.ncharged;
    int b[3], lo[3], hi[3];
    box_of_cta(prm, B, level, blockIdx.x / ncta, b, lo, hi);
    BoxShare share;
    bool handed = false;
    int nlist = -1;
    if (level < B.levels) {
        share = box_share<TIP_N, NC>(prm, B, level, b);
        handed = share_has_sums<TIP_N, NC>(share);
        if (handed && share.room > 0) nlist = *share_count<TIP_N, NC>(share);
    }
    const int nanc = handed ? B.levels - level : 0;
    const int ncand = nlist >= 0 ? nlist : nat, per = (ncand + ncta - 1) / ncta;
    const int first = min(rank * per, ncand), last = min(first + per, ncand);
    if (warp == 1 && lane <= nanc) pk.centre[lane] = box_centre(prm, B, level, b, lane);
    if (warp == 0 && lane < 3 * TIP_N) tip_node_table(prm, B, level, b, lane, s_node);
    if (tid >= 64 && tid < 64 + 6 * TIP_N) {
        const int i = tid - 64, a = i / (2 * TIP_N), c = i / TIP_N % 2, n = i % TIP_N;
        dfl x;
        if (box_child_node<TIP_N>(prm, B, level, a, a == 0 ? b[0] : (a == 1 ? b[1] : b[2]), c, n, x))
            cheb_row<TIP_N>(x, [&](int k, dfl w) { s_w[a][c][k][n] = w; });
    }
    __syncthreads();
    const bool on_nodes = tid < TIP_N3 / TIP_P;
    dfl p[3][TIP_P];
    TipSums S;
    S.zero();
    tip_nodes(s_node, tid, p);
    int nmid = 0, nzero = 0, place = -1, nleft = 0;
    for (int i0 = first; i0 < last; i0 += NT) {
        const int i = i0 + tid;
        int j0 = -1;
        if (i < last) {
            j0 = nlist >= 0 ? (int)*share_list<TIP_N, NC>(share, i) : i;
            box_gather(prm, tile + tid * FF_REC, j0);
            tip_limit(tile + tid * FF_REC);
        }
        box_pick<M_COUL, TIP_N, NT>(B, pk, level, nanc, tile, min(NT, last - i0), 1, true, nmid, nzero, place);
        if (place >= 0 && nleft + place < BOX_LEFT) s_left[nleft + place] = (unsigned short)j0;
        nleft += nzero;
        __syncthreads();
        for (int q = on_nodes ? 0 : nmid; q < nmid; q++) {
            const int j = pk.mid[q];
            tip_add<KIND, WITH_E, false>(p, tile[3 * j], tile[3 * j + 1], tile[3 * j + 2].z, S);
        }
        S.fold<WITH_E>();
        __syncthreads();
    }
    if (on_nodes) {
#pragma unroll
        for (int k = 0; k < K; k++)
#pragma unroll
            for (int i = 0; i < TIP_P; i++) own[k * TIP_N3 + TIP_P * tid + i] = S.get(k, i);
    }
    if (tid == 0) s_count = prm.natoms <= 65536 && nleft <= BOX_LEFT ? nleft : -1;
    cluster_meet();
    int before = 0, all = 0;
    for (int q = 0; q < ncta; q++) {
        const int n = cluster_ldi(cluster_addr(&s_count, q));
        if (q < rank) before += n;
        all = n < 0 || all < 0 ? -1 : all + n;
    }
    for (int i = tid; i < C4; i += NT) {  // two nodes
        float4 v = handed ? *share_cell(share, i) : make_float4(0.f, 0.f, 0.f, 0.f);
        for (int q = 0; q < ncta; q++) {
            const float4 o = cluster_ld4(cluster_addr(reinterpret_cast<const float4 *>(own) + i, q));
            const dfl s0 = df_add({v.x, v.y}, {o.x, o.y}), s1 = df_add({v.z, v.w}, {o.z, o.w});
            v = make_float4(s0.h, s0.l, s1.h, s1.l);
        }
        reinterpret_cast<float4 *>(sum)[i] = v;
    }
    cluster_meet();
    box_leave<TIP_N, NC, NT>(prm, B, level, b, s_left, nleft, before, all, rank == 0);
    dfl *ly = own;
    for (int q = rank; q < 8; q += ncta) {
        const int c[3] = {q >> 2, (q >> 1) & 1, q & 1}, ch[3] = {2 * b[0] + c[0], 2 * b[1] + c[1], 2 * b[2] + c[2]};
        if (!box_there(B, level - 1, ch)) continue;
        const BoxShare cs = box_share<TIP_N, NC>(prm, B, level - 1, ch);
        if (!share_has_sums<TIP_N, NC>(cs)) continue;
        auto along = [&](const dfl *v, int step, int axis, int n) -> dfl {  // at the child's node n
            dfl s = {0.f, 0.f};
#pragma unroll
            for (int k = 0; k < TIP_N; k++) df_fma(s, s_w[axis][c[axis]][k][n], v[k * step]);
            return two_sum(s.h, s.l);
        };
        for (int i = tid; i < K * TIP_N3; i += NT) lz[i] = along(sum + i / TIP_N * TIP_N, 1, 2, i % TIP_N);
        __syncthreads();
        for (int i = tid; i < K * TIP_N3; i += NT) ly[i] = along(lz + i / TIP_N2 * TIP_N2 + i % TIP_N, TIP_N, 1, i / TIP_N % TIP_N);
        __syncthreads();
        for (int i = tid; i < C4; i += NT) {
            const int k = i / (TIP_N3 / 2), r = i - k * (TIP_N3 / 2), x = r / (TIP_N2 / 2), yz = 2 * (r - x * (TIP_N2 / 2));
            const dfl s0 = along(ly + k * TIP_N3 + yz, TIP_N2, 0, x), s1 = along(ly + k * TIP_N3 + yz + 1, TIP_N2, 0, x);
            *share_cell(cs, i) = make_float4(s0.h, s0.l, s1.h, s1.l);
        }
        __syncthreads();
    }
}

// Leaves.  Shared memory: two atom tiles or the nodes' sums (then near atoms), the line and the plane.
template <bool WITH_E>
struct TipSmem {
    static constexpr int K = WITH_E ? 4 : 3, XS = BOX_S;
    static constexpr size_t tiles = sizeof(float4) * 2 * TIP_NT * FF_REC, nodes = sizeof(dfl) * K * TIP_N3;
    static constexpr size_t line = tiles > nodes ? tiles : nodes, plane = line + sizeof(dfl) * K * XS * TIP_N2;
    static constexpr size_t size = plane + sizeof(dfl) * K * TIP_X * XS * TIP_N;
};

template <int KIND, bool WITH_E, bool ORTHO>
__global__ void __launch_bounds__(TIP_NT, 2) tip_box_kernel(const __grid_constant__ FFParams prm, const __grid_constant__ BoxPrm B) {
    using Smem = TipSmem<WITH_E>;
    constexpr int K = Smem::K, NC = 2 * K, NT = TIP_NT, XS = Smem::XS, level = 0;  // NC: floats of a node
    extern __shared__ __align__(128) unsigned char tip_raw[];
    float4 *tiles = reinterpret_cast<float4 *>(tip_raw);
    dfl *line = reinterpret_cast<dfl *>(tip_raw + Smem::line);    // [K][x][10][10]
    dfl *plane = reinterpret_cast<dfl *>(tip_raw + Smem::plane);  // [K][x - xh][y][10]
    __shared__ BoxNear s_near;
    __shared__ BoxPick<NT> pk;
    __shared__ dfl s_node[3][TIP_N][3], s_pt[3][BOX_S][3];                // parts of the nodes' and the points' positions
    __shared__ dfl s_wx[XS][TIP_N], s_wy[XS][TIP_N], s_wz[XS][TIP_N];

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nat = prm.ncharged;
    int b[3], lo[3], hi[3];
    box_of_cta(prm, B, level, blockIdx.x, b, lo, hi);
    BoxShare share;
    bool handed = false;
    int nlist = -1;
    if (level < B.levels) {
        share = box_share<TIP_N, NC>(prm, B, level, b);
        handed = share_has_sums<TIP_N, NC>(share);
        if (handed && share.room > 0) nlist = *share_count<TIP_N, NC>(share);
    }
    const int nanc = handed ? B.levels - level : 0;
    const int ncand = nlist >= 0 ? nlist : nat;
    // ---- tables of this box
    if (warp == 1 && lane <= nanc) pk.centre[lane] = box_centre(prm, B, level, b, lane);
    if (warp == 0 && lane < 3 * TIP_N) tip_node_table(prm, B, level, b, lane, s_node);
    if (tid >= 64 && tid < 64 + 48) {
        const int a = (tid - 64) >> 4, j = (tid - 64) & 15;
        const float g = (float)(prm.i0[a] + (a == 0 ? lo[0] : (a == 1 ? lo[1] : lo[2])) + j);
#pragma unroll
        for (int k = 0; k < 3; k++) s_pt[a][j][k] = df_mul_f(B.step[a][k], g);
    }
    for (int i = tid; i < 3 * XS * TIP_N; i += NT) {
        const int a = i / (XS * TIP_N), pt = (i / TIP_N) % XS, k = i % TIP_N;
        const int m = (a == 0 ? hi[0] - lo[0] : (a == 1 ? hi[1] - lo[1] : hi[2] - lo[2])) + 1;
        (a == 0 ? s_wx : (a == 1 ? s_wy : s_wz))[pt][k] = {cheb_points<TIP_N>().w[m][pt][k], c_points_low.w[m][pt][k]};
    }
    __syncthreads();

    // ---- far charges on the nodes: a thread has four
    const bool on_nodes = tid < TIP_N3 / TIP_P;
    dfl p[3][TIP_P];
    TipSums S;
    S.zero();
    tip_nodes(s_node, tid, p);
    const bool wide = nat > 65536;
    const int near_cap = wide ? BOX_NEAR / 2 : BOX_NEAR;
    auto near_at = [&](int i) -> int { return s_near.at(wide, i); };
    int nmid = 0, nzero = 0, place = -1, nnear = 0;
    auto gather = [&](int t, bool all) -> int {  // as in ff_box_kernel
        const int i = t * NT + tid;
        int j = -1;
        if (i < (all ? nat : ncand)) {
            j = all || nlist < 0 ? i : (int)*share_list<TIP_N, NC>(share, i);
            box_gather(prm, tiles + ((t & 1) * NT + tid) * FF_REC, j);
            tip_limit(tiles + ((t & 1) * NT + tid) * FF_REC);
        }
        return j;
    };
    for (int t = 0; t < (ncand + NT - 1) / NT; t++) {
        const float4 *T = tiles + (t & 1) * NT * FF_REC;
        const int j0 = gather(t, false);
        box_pick<M_COUL, TIP_N, NT>(B, pk, level, nanc, T, min(NT, ncand - t * NT), 1, true, nmid, nzero, place);
        if (place >= 0 && nnear + place < near_cap) s_near.set(wide, nnear + place, j0);
        nnear += nzero;
        __syncthreads();
        for (int i = on_nodes ? 0 : nmid; i < nmid; i++) {
            const int j = pk.mid[i];
            tip_add<KIND, WITH_E, false>(p, T[3 * j], T[3 * j + 1], T[3 * j + 2].z, S);
        }
        S.fold<WITH_E>();
        __syncthreads();
    }
    // ---- the nodes' sums and the parent's interpolated sums
    dfl *nodes = reinterpret_cast<dfl *>(tiles);  // [K][10][10][10]
    if (on_nodes) {
#pragma unroll
        for (int k = 0; k < K; k++) {
            dfl v[TIP_P];
#pragma unroll
            for (int i = 0; i < TIP_P; i++) v[i] = S.get(k, i);
            if (handed) {
#pragma unroll
                for (int e = 0; e < 2; e++) {
                    const float4 o = *share_cell(share, k * (TIP_N3 / 2) + 2 * tid + e);
                    v[2 * e] = df_add(v[2 * e], {o.x, o.y});
                    v[2 * e + 1] = df_add(v[2 * e + 1], {o.z, o.w});
                }
            }
#pragma unroll
            for (int i = 0; i < TIP_P; i++) nodes[k * TIP_N3 + TIP_P * tid + i] = v[i];
        }
    }
    __syncthreads();
    // ---- along x, a thread one node and every other x
    for (int i = tid; i < 2 * K * TIP_N2; i += NT) {
        const int x0 = i / (K * TIP_N2), q = i - x0 * (K * TIP_N2), k = q / TIP_N2, r = q - k * TIP_N2;
        dfl v[TIP_N];
#pragma unroll
        for (int a = 0; a < TIP_N; a++) v[a] = nodes[k * TIP_N3 + a * TIP_N2 + r];
#pragma unroll 1
        for (int x = x0; x < XS; x += 2) {
            dfl s = {0.f, 0.f};
#pragma unroll
            for (int a = 0; a < TIP_N; a++) df_fma(s, s_wx[x][a], v[a]);
            line[(k * XS + x) * TIP_N2 + r] = two_sum(s.h, s.l);
        }
    }
    __syncthreads();
    auto stage = [&](int first, int last) {  // near atoms into the tiles' space
        for (int i = tid; i < (last - first) * FF_REC; i += NT)
            tiles[i] = ldg4(prm.atoms + (size_t)near_at(first + i / FF_REC) * FF_REC + i % FF_REC);
        __syncthreads();
    };
    const bool listed = nnear <= near_cap, staged = nnear <= BOX_STAGE;
    if (listed && staged) stage(0, nnear);
    const int mx = hi[0] - lo[0] + 1, my = hi[1] - lo[1] + 1, mz = hi[2] - lo[2] + 1;
#pragma unroll 1
    for (int xh = 0; xh < mx; xh += TIP_X) {
        // ---- along y, for four of the box's x
        __syncthreads();  // the runs of the four before have read the plane
        for (int i = tid; i < K * TIP_X * XS * TIP_N; i += NT) {
            const int c = i % TIP_N, y = i / TIP_N % XS, x = i / (TIP_N * XS) % TIP_X, k = i / (TIP_N * XS * TIP_X);
            dfl s = {0.f, 0.f};
#pragma unroll
            for (int a = 0; a < TIP_N; a++) df_fma(s, s_wy[y][a], line[(k * XS + xh + x) * TIP_N2 + a * TIP_N + c]);
            plane[i] = two_sum(s.h, s.l);
        }
        __syncthreads();
        const int nrun = min(TIP_X, mx - xh) * my * 4;
#pragma unroll 1
        for (int c0 = 0; c0 < nrun; c0 += NT) {
            const int c = min(c0 + tid, nrun - 1);  // threads past the end repeat the last run and store nothing
            const int h = c & 3, xy = c >> 2, x = xy / my, y = xy - x * my;
            // ---- along z, every fourth point from h
            S.zero();
#pragma unroll
            for (int k = 0; k < K; k++) {
                const dfl *v = plane + ((k * TIP_X + x) * XS + y) * TIP_N;
#pragma unroll
                for (int i = 0; i < TIP_P; i++) {
                    dfl s = {0.f, 0.f};
                    const dfl *w = s_wz[h + 4 * i];
#pragma unroll
                    for (int a = 0; a < TIP_N; a++) df_fma(s, w[a], v[a]);
                    s = two_sum(s.h, s.l);
                    if (k == 3) S.E[i] = s;
                    else S.F[k < 3 ? k : 0][i] = s;
                }
            }
#pragma unroll
            for (int k = 0; k < 3; k++) {
                const dfl q = df_add(s_pt[0][xh + x][k], s_pt[1][y][k]);
#pragma unroll
                for (int i = 0; i < TIP_P; i++)
                    if (k == 2 || i == 0 || !ORTHO) p[k][i] = df_add(q, s_pt[2][h + 4 * i][k]);
            }
            if (listed) {
                for (int n0 = 0; n0 < nnear; n0 += BOX_STAGE) {
                    const int n1 = min(nnear, n0 + BOX_STAGE);
                    if (!staged) stage(n0, n1);
                    for (int j = 0; j < n1 - n0; j++)
                        tip_add<KIND, WITH_E, ORTHO>(p, tiles[3 * j], tiles[3 * j + 1], tiles[3 * j + 2].z, S);
                    if (!staged) __syncthreads();
                }
            } else {  // more near atoms than the list holds: through all atoms again
                for (int t = 0; t < (nat + NT - 1) / NT; t++) {
                    const float4 *T = tiles + (t & 1) * NT * FF_REC;
                    gather(t, true);
                    box_pick<M_COUL, TIP_N, NT>(B, pk, level, nanc, T, min(NT, nat - t * NT), 0, true, nmid, nzero, place);
                    __syncthreads();
                    for (int i = 0; i < nmid; i++) {
                        const int j = pk.mid[i];
                        tip_add<KIND, WITH_E, ORTHO>(p, T[3 * j], T[3 * j + 1], T[3 * j + 2].z, S);
                    }
                    __syncthreads();
                }
            }
            S.fold<WITH_E>();
            if (c0 + tid >= nrun) continue;
            float4 *dst = prm.FE + ((long long)(lo[0] + xh + x) * prm.ns[1] + lo[1] + y) * prm.ns[2] + lo[2] + h;
#pragma unroll
            for (int i = 0; i < TIP_P; i++) {
                if (h + 4 * i >= mz) break;
                tip_store<KIND, WITH_E>(prm, S, i, dst + 4 * i);
            }
        }
    }
}

// ----------------------------------------------------------------------------- host

template <int KIND, bool WITH_E, bool ORTHO>
static int launch_tip_boxes(const FFParams &prm, BoxPrm B, cudaStream_t st) {
    constexpr int up = (int)TipUpSmem<WITH_E>::size, leaf = (int)TipSmem<WITH_E>::size;
    PPGPU_CUDA(cudaFuncSetAttribute(tip_up_kernel<KIND, WITH_E>, cudaFuncAttributeMaxDynamicSharedMemorySize, up), "tip boxes' shared memory");
    PPGPU_CUDA(cudaFuncSetAttribute(tip_box_kernel<KIND, WITH_E, ORTHO>, cudaFuncAttributeMaxDynamicSharedMemorySize, leaf),
               "tip boxes' shared memory");
    for (B.level = B.levels; B.level >= 0; B.level--) {
        long long n = 1;
        for (int k = 0; k < 3; k++) n *= ((B.nb[k] - 1) >> B.level) + 1;
        if (n > 0x0fffffffLL) return set_error(PPGPU_ERR_ARG, "ff grid too large (%lld boxes)", n);
        if (B.level > 0) {
            int rc = launch_box_up(tip_up_kernel<KIND, WITH_E>, up, n, prm, B, st);
            if (rc) return rc;
        } else {
            tip_box_kernel<KIND, WITH_E, ORTHO><<<(unsigned)n, TIP_NT, leaf, st>>>(prm, B);
            PPGPU_CHECK_LAUNCH("tip_box_kernel launch");
        }
    }
    return set_ok();
}

// Grids and charges summed by boxes.  dz2, pair by pair against by boxes, at 0.1 A steps (in brackets
// 0.3 A where it differs): 200^3 points (2197 leaves), 342 charges 16.7 against 1.86 ms, 60: 3.02 against
// 1.33; 140^3 (729) 342: 5.85 against 1.29, 60: 1.07 against 0.67 (0.75), 30: 0.55 against 0.41 (0.45), 6: 0.15
// against 0.19; 96^3 (216) 342: 1.98 against 1.03, 90: 0.54 against 0.51 (0.71), 60: 0.38 against 0.39 (0.52);
// 64^3 (64 leaves) 342: 0.69 against 0.83, the boxes too few for 152 SMs.
//   Levels above the leaves, 0, 1 and 2: 140^3, 90 charges 0.92, 0.94, 0.98 ms (6.6e4 charge-boxes), 96^3, 342 1.22, 1.03,
// 1.06 (7.4e4), 140^3, 540 3.69, 1.94, 1.99 (3.9e5), 200^3, 342 6.6, 2.15, 1.86 (7.5e5).
//   Flat and narrow grids, whose leaves have few points for the 1000 nodes, or no room for what is handed to them (pair by
// pair against by boxes): 990x1x547, 138 charges 0.39 against 3.1 ms, 2x319x1251, 567 2.5 against 9.0, 4x613x123, 585 1.35 against
// 3.1.  Of 900 calls (half of them flat or narrow) 3 are slower by boxes than pair by pair, by 1.3 times.
static bool tip_box_rule(const FFParams &prm, bool with_e, BoxPrm *B) {
    const double boxes = box_count(prm), work = prm.ncharged * boxes, need = 15.0 + 20000.0 / boxes;
    if (!(boxes >= 200 && prm.ncharged >= need)) return false;  // before planning, which small calls would feel
    double H;
    box_plan(prm, TIP_N, TIP_KAPPA, TIP_H, B, &H);
    B->levels = prm.accumulate || work < 7e4 ? 0 : (work < 5e5 ? 1 : (work < 1e8 ? 2 : 3));
    const double leaf = box_leaf(*B);
    if (leaf < (B->levels == 0 ? 1024 : (with_e ? 2000 : 1500))) return false;
    return H * TIP_KAPPA <= 36.0 && prm.ncharged >= need * std::max(1.0, 2500.0 / leaf);
}

FFRoute ff_tip_route(const FFParams &prm, bool with_e) {
    BoxPrm B;
    return tip_box_rule(prm, with_e, &B) ? FFRoute{TIP_N, B.levels} : FFRoute{0, 0};
}

template <int KIND, bool WITH_E, bool ORTHO>
static int launch_tip(FFParams &prm, cudaStream_t st) {
    BoxPrm B;
    if (tip_box_rule(prm, WITH_E, &B)) return launch_tip_boxes<KIND, WITH_E, ORTHO>(prm, B, st);
    prm.nzc = (prm.ns[2] + TIP_P - 1) / TIP_P;
    prm.nchunks = (long long)prm.ns[0] * prm.ns[1] * prm.nzc;
    const long long nblk = (prm.nchunks + TIP_THREADS - 1) / TIP_THREADS;
    if (nblk <= 0) return set_ok();
    if (nblk > 0x7fffffffLL) return set_error(PPGPU_ERR_ARG, "ff grid too large (%lld blocks)", nblk);
    ff_tip_kernel<KIND, WITH_E, ORTHO><<<(unsigned)nblk, TIP_THREADS, 0, st>>>(prm);
    PPGPU_CHECK_LAUNCH("ff_tip_kernel launch");
    return set_ok();
}

template <int KIND>
static int launch_tip_kind(FFParams &prm, bool with_e, bool ortho, cudaStream_t st) {
    if (with_e) return ortho ? launch_tip<KIND, true, true>(prm, st) : launch_tip<KIND, true, false>(prm, st);
    return ortho ? launch_tip<KIND, false, true>(prm, st) : launch_tip<KIND, false, false>(prm, st);
}

int launch_ff_tip(FFParams &prm, int kind, bool with_e, bool ortho, cudaStream_t st) {
    return kind == 1 ? launch_tip_kind<1>(prm, with_e, ortho, st) : launch_tip_kind<2>(prm, with_e, ortho, st);
}

}  // namespace ppgpu
