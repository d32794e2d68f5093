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
//   342 charges on 200^3 points: dz2 423 ms in float64, 16.7 ms pair by pair here, 2.44 by boxes (error
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
        for (int i = tid; i < nj * FF_REC; i += TIP_THREADS) s_at[i] = prm.atoms[(size_t)base * FF_REC + i];
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
// (R >= 9 H + h) are summed on 8^3 nodes, which with the smoother Coulomb terms leaves 6e-10 of a
// pair's field, a hundredth of the stored value's rounding; nodes, weights and sums are
// double-floats.  256 threads: for the nodes 128 halves of a node column x 2 parts of the atoms,
// for the points runs of every fourth point of a column (neighbours write neighbouring points).
// The interpolation goes along x (line), then along y for half of the box's x at a time (plane),
// then along z into a run's sums.  128 registers, two CTAs a SM.

constexpr double TIP_KAPPA = 9.0;
constexpr int TIP_NT = 256;

// acc += w v (both double-floats).
__device__ __forceinline__ void df_fma(dfl &acc, dfl w, dfl v) { df_acc(acc, df_mul_raw(w, v)); }

template <bool WITH_E>
constexpr size_t tip_box_smem() {
    return sizeof(float4) * 2 * TIP_NT * FF_REC + 2 * sizeof(dfl) * (WITH_E ? 4 : 3) * BOX_S * 64;
}

template <int KIND, bool WITH_E, bool ORTHO, bool LEAF>
__global__ void __launch_bounds__(TIP_NT, 2) tip_box_kernel(const __grid_constant__ FFParams prm, const __grid_constant__ BoxPrm B) {
    constexpr int K = WITH_E ? 4 : 3, NC = 2 * K, NT = TIP_NT;  // components; floats of a node
    extern __shared__ __align__(128) unsigned char tip_raw[];
    float4 *tiles = reinterpret_cast<float4 *>(tip_raw);                                   // atoms; the nodes' sums; near atoms
    dfl *line = reinterpret_cast<dfl *>(tip_raw + sizeof(float4) * 2 * NT * FF_REC);      // [K][x][8][8]
    dfl *plane = line + K * BOX_S * 64;                                                    // [K][8 of x][y][8]; parts of the nodes' sums
    __shared__ unsigned short s_near[LEAF ? BOX_NEAR : 1];
    __shared__ unsigned short s_left[NT];
    __shared__ BoxPick<NT> pk;
    __shared__ dfl s_node[3][BOX_N][3], s_pt[3][BOX_S][3];                // parts of the nodes' and the points' positions
    __shared__ dfl s_wx[BOX_S][BOX_N], s_wy[BOX_S][BOX_N], s_wz[BOX_S][BOX_N];

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int level = LEAF ? 0 : B.level, nat = prm.ncharged;
    int b[3], lo[3], hi[3];
    box_of_cta(prm, B, level, b, lo, hi);
    BoxShare share;
    bool handed = false;
    int nlist = -1;
    if (level < B.levels) {
        share = box_share<NC>(prm, B, level, b);
        handed = share_has_slot<NC>(share, level);
        if (handed && share.room > 0) nlist = *share_count(share, level);
    }
    const int nanc = handed ? B.levels - level : 0;
    const int ncand = nlist >= 0 ? nlist : nat;
    // ---- tables of this box
    if (warp == 1 && lane <= nanc) pk.centre[lane] = box_centre(prm, B, level, b, lane);
    if (warp == 0 && lane < 24) {
        const int a = lane >> 3, i = lane & 7;
        int l, h;
        box_span(prm, B, level, a, a == 0 ? b[0] : (a == 1 ? b[1] : b[2]), l, h);
        const dfl g = df_add(df_mul_f(cheb_t(i), box_half(l, h)), {0.5f * (float)(l + h) + (float)prm.i0[a], 0.f});
#pragma unroll
        for (int k = 0; k < 3; k++) s_node[a][i][k] = df_mul(B.step[a][k], g);
    }
    if (LEAF && tid >= 64 && tid < 64 + 48) {
        const int a = (tid - 64) >> 4, j = (tid - 64) & 15;
        const float g = (float)(prm.i0[a] + (a == 0 ? lo[0] : (a == 1 ? lo[1] : lo[2])) + j);
#pragma unroll
        for (int k = 0; k < 3; k++) s_pt[a][j][k] = df_mul_f(B.step[a][k], g);
    }
    for (int i = tid; i < 3 * BOX_S * BOX_N; i += NT) {
        const int a = i / (BOX_S * BOX_N), pt = (i / BOX_N) % BOX_S, k = i % BOX_N;
        dfl w;
        if constexpr (LEAF) {
            const int m = (a == 0 ? hi[0] - lo[0] : (a == 1 ? hi[1] - lo[1] : hi[2] - lo[2])) + 1;
            w = {c_cheb_points.w[m][pt][k], c_cheb_points.l[m][pt][k]};
        } else {
            w = box_child_weight(prm, B, level, a, a == 0 ? b[0] : (a == 1 ? b[1] : b[2]), pt, k);
        }
        (a == 0 ? s_wx : (a == 1 ? s_wy : s_wz))[pt][k] = w;
    }
    __syncthreads();

    // ---- far charges on the nodes: thread = half of a node column, one of two parts of the atoms
    const int sub = tid >> 7, col = (tid & 127) >> 1, half = tid & 1;
    dfl p[3][TIP_P];
    TipSums S;
    S.zero();
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const dfl xy = df_add(s_node[0][col >> 3][k], s_node[1][col & 7][k]);
#pragma unroll
        for (int i = 0; i < TIP_P; i++)
            if (k == 2 || i == 0 || !ORTHO) p[k][i] = df_add(xy, s_node[2][4 * half + i][k]);
    }
    const bool wide = nat > 65536;
    const int near_cap = wide ? BOX_NEAR / 2 : BOX_NEAR;
    auto near_at = [&](int i) -> int { return wide ? reinterpret_cast<const int *>(s_near)[i] : (int)s_near[i]; };
    int nmid = 0, nzero = 0, place = -1, nnear = 0;
    auto gather = [&](int t, bool all) -> int {  // as in ff_box_kernel
        const int i = t * NT + tid;
        int j = -1;
        if (i < (all ? nat : ncand)) {
            j = all || nlist < 0 ? i : (int)*share_list(share, level, i);
            box_gather(prm, tiles + ((t & 1) * NT + tid) * FF_REC, j);
        }
        return j;
    };
    for (int t = 0; t < (ncand + NT - 1) / NT; t++) {
        const float4 *T = tiles + (t & 1) * NT * FF_REC;
        const int j0 = gather(t, false);
        box_pick<M_COUL, NT>(B, pk, level, nanc, T, min(NT, ncand - t * NT), 1, true, nmid, nzero, place);
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
        for (int i = sub; i < nmid; i += 2) {
            const int j = pk.mid[i];
            tip_add<KIND, WITH_E, ORTHO>(p, T[3 * j], T[3 * j + 1], T[3 * j + 2].z, S);
        }
        S.fold<WITH_E>();
        __syncthreads();
    }
    if constexpr (!LEAF) box_leave_count<NC>(prm, B, level, b, nnear);
    // ---- the nodes' sums: both parts of the atoms and the parent's interpolated sums
    dfl *nodes = reinterpret_cast<dfl *>(tiles);  // [K][8][8][8]
    if (sub == 1) {
#pragma unroll
        for (int k = 0; k < K; k++)
#pragma unroll
            for (int i = 0; i < TIP_P; i++) plane[(k * TIP_P + i) * 128 + (tid & 127)] = S.get(k, i);
    }
    __syncthreads();
    if (sub == 0) {
#pragma unroll
        for (int k = 0; k < K; k++) {
            dfl v[TIP_P];
#pragma unroll
            for (int i = 0; i < TIP_P; i++) v[i] = df_add(S.get(k, i), plane[(k * TIP_P + i) * 128 + tid]);
            if (handed) {
#pragma unroll
                for (int e = 0; e < 2; e++) {
                    const float4 o = *share_slot<NC>(share, level, k * 256 + col * 4 + half * 2 + e);
                    v[2 * e] = df_add(v[2 * e], {o.x, o.y});
                    v[2 * e + 1] = df_add(v[2 * e + 1], {o.z, o.w});
                }
            }
#pragma unroll
            for (int i = 0; i < TIP_P; i++) nodes[k * BOX_N3 + col * 8 + half * 4 + i] = v[i];
        }
    }
    __syncthreads();
    // ---- along x
    if (tid < K * 64) {
        const int k = tid >> 6, r = tid & 63;
        dfl v[BOX_N];
#pragma unroll
        for (int a = 0; a < BOX_N; a++) v[a] = nodes[k * BOX_N3 + a * 64 + r];
#pragma unroll 1
        for (int x = 0; x < BOX_S; x++) {
            dfl s = {0.f, 0.f};
#pragma unroll
            for (int a = 0; a < BOX_N; a++) df_fma(s, s_wx[x][a], v[a]);
            line[(k * BOX_S + x) * 64 + r] = two_sum(s.h, s.l);
        }
    }
    __syncthreads();
    auto stage = [&](int first, int last) {  // near atoms into the tiles' space
        for (int i = tid; i < (last - first) * FF_REC; i += NT)
            tiles[i] = ldg4(prm.atoms + (size_t)near_at(first + i / FF_REC) * FF_REC + i % FF_REC);
        __syncthreads();
    };
    const bool listed = nnear <= near_cap, staged = nnear <= BOX_STAGE;
    if (LEAF && listed && staged) stage(0, nnear);
    const int mx = LEAF ? hi[0] - lo[0] + 1 : BOX_S, my = LEAF ? hi[1] - lo[1] + 1 : BOX_S, mz = hi[2] - lo[2] + 1;
#pragma unroll 1
    for (int xh = 0; xh < mx; xh += 8) {
        // ---- along y, for eight of the box's x
        __syncthreads();  // the runs of the eight before have read the plane
        for (int i = tid; i < K * 8 * 16 * 8; i += NT) {
            const int c = i & 7, y = (i >> 3) & 15, x = (i >> 7) & 7, k = i >> 10;
            dfl s = {0.f, 0.f};
#pragma unroll
            for (int a = 0; a < BOX_N; a++) df_fma(s, s_wy[y][a], line[(k * BOX_S + xh + x) * 64 + a * 8 + c]);
            plane[i] = two_sum(s.h, s.l);
        }
        __syncthreads();
        const int nrun = min(8, mx - xh) * my * 4;
#pragma unroll 1
        for (int c0 = 0; c0 < nrun; c0 += NT) {
            const int c = min(c0 + tid, nrun - 1);  // threads past the end repeat the last run and store nothing
            const int h = c & 3, xy = c >> 2, x = xy / my, y = xy - x * my;
            // ---- along z: leaves every fourth point from h, upper boxes four nodes of a child
            S.zero();
#pragma unroll
            for (int k = 0; k < K; k++) {
                const dfl *v = plane + ((k * 8 + x) * 16 + y) * 8;
#pragma unroll
                for (int i = 0; i < TIP_P; i++) {
                    dfl s = {0.f, 0.f};
                    const dfl *w = s_wz[LEAF ? h + 4 * i : 4 * h + i];
#pragma unroll
                    for (int a = 0; a < BOX_N; a++) df_fma(s, w[a], v[a]);
                    s = two_sum(s.h, s.l);
                    if (k == 3) S.E[i] = s;
                    else S.F[k < 3 ? k : 0][i] = s;
                }
            }
            if constexpr (!LEAF) {
                const int ch[3] = {2 * b[0] + ((xh + x) >> 3), 2 * b[1] + (y >> 3), 2 * b[2] + (h >> 1)};
                if (!box_there(B, level - 1, ch)) continue;
                const BoxShare cs = box_share<NC>(prm, B, level - 1, ch);
                if (!share_has_slot<NC>(cs, level - 1)) continue;
#pragma unroll
                for (int k = 0; k < K; k++)
#pragma unroll
                    for (int e = 0; e < 2; e++) {
                        const dfl u = S.get(k, 2 * e), w = S.get(k, 2 * e + 1);
                        *share_slot<NC>(cs, level - 1, k * 256 + (((xh + x) & 7) * 8 + (y & 7)) * 4 + (h & 1) * 2 + e) =
                            make_float4(u.h, u.l, w.h, w.l);
                    }
            } else {
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
                        box_pick<M_COUL, NT>(B, pk, level, nanc, T, min(NT, nat - t * NT), 0, true, nmid, nzero, place);
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
}

// ----------------------------------------------------------------------------- host

template <int KIND, bool WITH_E, bool ORTHO>
static int launch_tip_boxes(const FFParams &prm, BoxPrm B, cudaStream_t st) {
    constexpr int smem = (int)tip_box_smem<WITH_E>();
    PPGPU_CUDA(cudaFuncSetAttribute(tip_box_kernel<KIND, WITH_E, ORTHO, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem),
               "tip boxes' shared memory");
    PPGPU_CUDA(cudaFuncSetAttribute(tip_box_kernel<KIND, WITH_E, ORTHO, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem),
               "tip boxes' shared memory");
    for (B.level = B.levels; B.level >= 0; B.level--) {
        long long n = 1;
        for (int k = 0; k < 3; k++) n *= ((B.nb[k] - 1) >> B.level) + 1;
        if (n > 0x7fffffffLL) return set_error(PPGPU_ERR_ARG, "ff grid too large (%lld boxes)", n);
        if (B.level > 0)
            tip_box_kernel<KIND, WITH_E, ORTHO, false><<<(unsigned)n, TIP_NT, smem, st>>>(prm, B);
        else
            tip_box_kernel<KIND, WITH_E, ORTHO, true><<<(unsigned)n, TIP_NT, smem, st>>>(prm, B);
    }
    PPGPU_CHECK_LAUNCH("tip_box_kernel launch");
    return set_ok();
}

// Grids and charges summed by boxes.  dz2, pair by pair against by boxes (0.05 to 0.3 A steps alike
// where not given): 200^3 points, 342 charges 16.7 against 2.44 ms (3.49 without the level above);
// 140^3 (729 leaves) 342: 5.84 against 1.95, 90: 1.57 against 0.60, 60: 1.06 against 0.63 (0.05 A) to
// 1.00 (0.3 A), 30: 0.55 against 0.44 to 0.55; 96^3 (216 leaves) 90: 0.54 against 0.45, 60: 0.37
// against 0.38 to 0.51; 64^3 (64 leaves) 342: 0.68 against 1.0 to 1.5, the boxes too few for 152 SMs.
// A level above the leaves: 342 charges gain at 2197 leaves, not at 729 (2.5e5 charge-boxes).
static bool tip_box_rule(const FFParams &prm, double H, BoxPrm *B) {
    const double boxes = (double)B->nb[0] * B->nb[1] * B->nb[2], work = prm.ncharged * boxes;
    B->levels = prm.accumulate || work < 4e5 ? 0 : (work < 1e8 ? 1 : 2);
    return boxes >= 200 && H <= 5.0 && prm.ncharged >= 40.0 + 10000.0 / boxes;
}

template <int KIND, bool WITH_E, bool ORTHO>
static int launch_tip(FFParams &prm, cudaStream_t st) {
    BoxPrm B;
    double H;
    box_plan(prm, TIP_KAPPA, TIP_H, &B, &H);
    if (tip_box_rule(prm, H, &B)) return launch_tip_boxes<KIND, WITH_E, ORTHO>(prm, B, st);
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
