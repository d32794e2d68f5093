// pp_relax.cu -- probe-particle relaxation on sm_103a.
//
// CPU-core semantics (ppafm/cpp/ProbeParticle.cpp):
//   relaxTipStrokes_omp 682-701, relaxTipStroke 633-676, relaxProbe 297-313,
//   getPPforce 282-294, FIREstate::move 142-174, RELAX::move 84-88,
//   interpolate3DvecWrap + SET_GRID_IND (ppafm/cpp/Grid.h:66-69, 93-111),
//   forceRSpring (ppafm/cpp/Forces.h:85-89);
//   Fz2df (ppafm/common.py:421-430) fused as a per-pixel epilogue.
// AFMulator semantics (ppafm/ocl/cl/relax.cl):
//   relaxStrokesTilted 391-464, update_FIRE 105-126, tipForce 37-41, convolveZ 571-608.
//
// Design (GB300):
//  * One lane per stroke (pixel column), or one per axis of a stroke on scans too small to fill
//    the GPU (relax_axis_kernel).  A lane's whole z-walk is a single flattened loop in which
//    every trip interpolates the force once (8 x 16-byte __ldg of the interleaved float4 grid;
//    scans of one wave only when the probe has left its cell), so lanes that converge early at one height move on to
//    their next height instead of idling; the warp leaves the loop on a vote once all of its
//    lanes have finished their strokes.
//  * Precision, chosen by measurement against the float64 reference on a GB300, whose
//    float64 rate is 1/64 of its float32 rate: the probe displacement d = r - r_tip, the grid
//    coordinate, the trilinear weights and interpolation sum, the springs and the force sum
//    are double-float (pp_df.cuh: two floats, ~48 significant bits); the FIRE state
//    (velocity, dt, mixing coefficient) and the residual force it consumes are float32.
//    Rounding noise in the interpolated force of ~3e-8 relative (plain float32) moves the
//    stopping point of a few pixel heights in 1e5 by more than 1e-3 A inside the
//    |F| < 1e-4 eV/A ball (the soft lateral spring leaves it ~6e-3 A wide); 1e-9 relative
//    noise moves none, and neither does a float32 FIRE state.  The only difference from the
//    reference left is the float32 storage of the grid values.  Float64 is used once per
//    height (tip grid coordinate), not per iteration.
//  * Trilinear weights are explicit (no texture filtering).
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "pp_axis_lanes.cuh"
#include "pp_common.cuh"
#include "pp_df.cuh"
#include "pp_relax_dev.cuh"

namespace ppgpu {

struct StrokeIO {  // relaxTipStrokes semantics (float64 in/out)
    int nstroke, nstep;
    const double *rTips;
    double *rs, *fs;
    int *iters, *itrsum;
};

struct ScanIO {  // regular scan semantics
    int nx, ny, nz;
    const double *xs, *ys, *zs;
    double off[3];
    dfl offd[3];
    float *fzs, *ppos, *df;
    int *iters;
    int nw;
    float W[MAX_DF_TAPS];
};

// The corners of the cell that a stroke was in last, all four channels (Corners' AFMulator form).
struct Corners4 {
    long long cell = -1;
    float4 c[8];
};

// The same as interp_force_df, all four channels, at a float grid coordinate (AFMulator path); KEEP:
// gathering when the stroke has left its cell.
template <bool KEEP>
__device__ __forceinline__ float4 interp_fe4(const float4 *__restrict__ FE, int n0, int n1, int n2, float3 g, Corners4 &K) {
    const float fx = floorf(g.x), fy = floorf(g.y), fz = floorf(g.z);
    const float tx = g.x - fx, ty = g.y - fy, tz = g.z - fz;
    const float mx = 1.f - tx, my = 1.f - ty, mz = 1.f - tz;
    const int ix0 = wrap_index((int)fx, n0), iy0 = wrap_index((int)fy, n1), iz0 = wrap_index((int)fz, n2);
    float4 *c = K.c;
    if (!KEEP) {
        const int ix1 = (ix0 + 1 == n0) ? 0 : ix0 + 1;
        const int iy1 = (iy0 + 1 == n1) ? 0 : iy0 + 1;
        const int iz1 = (iz0 + 1 == n2) ? 0 : iz0 + 1;
        const long long r00 = ((long long)ix0 * n1 + iy0) * n2, r01 = ((long long)ix0 * n1 + iy1) * n2;
        const long long r10 = ((long long)ix1 * n1 + iy0) * n2, r11 = ((long long)ix1 * n1 + iy1) * n2;
        c[0] = ldg4(FE + r00 + iz0), c[1] = ldg4(FE + r00 + iz1);
        c[2] = ldg4(FE + r01 + iz0), c[3] = ldg4(FE + r01 + iz1);
        c[4] = ldg4(FE + r10 + iz0), c[5] = ldg4(FE + r10 + iz1);
        c[6] = ldg4(FE + r11 + iz0), c[7] = ldg4(FE + r11 + iz1);
    } else {
        const long long cell = ((long long)ix0 * n1 + iy0) * n2 + iz0;
        if (cell != K.cell) {
            K.cell = cell;
            const long long dx = ix0 + 1 == n0 ? -(long long)ix0 * n1 * n2 : (long long)n1 * n2;
            const long long dy = iy0 + 1 == n1 ? -(long long)iy0 * n2 : (long long)n2;
            const int dz = iz0 + 1 == n2 ? -iz0 : 1;
#pragma unroll
            for (int k = 0; k < 8; k++) c[k] = ldg4(FE + cell + ((k & 4) ? dx : 0) + ((k & 2) ? dy : 0) + ((k & 1) ? dz : 0));
        }
    }
    float4 o;
#define PP_LERP3(a)                                                                                \
    {                                                                                              \
        const float v00 = fmaf(c[4].a, tx, c[0].a * mx), v10 = fmaf(c[6].a, tx, c[2].a * mx);     \
        const float v01 = fmaf(c[5].a, tx, c[1].a * mx), v11 = fmaf(c[7].a, tx, c[3].a * mx);     \
        const float v0 = fmaf(v10, ty, v00 * my), v1 = fmaf(v11, ty, v01 * my);                   \
        o.a = fmaf(v1, tz, v0 * mz);                                                               \
    }
    PP_LERP3(x) PP_LERP3(y) PP_LERP3(z) PP_LERP3(w)
#undef PP_LERP3
    return o;
}

// --------------------------------------------------------- CPU-core semantics

// Scan mode keeps a per-height table in shared memory, so that a height change needs no float64:
// z and g_z = dic . (0, 0, z) as double-floats; with a diagonal metric only z's own grid coordinate
// changes, and the table holds its cell and fraction instead.
constexpr int ZTAB = 4;

__device__ __forceinline__ void fill_ztab(dfl *ztab, const RelaxPrm &P, const double *zs, int nz) {
    for (int i = threadIdx.x; i < nz; i += RELAX_THREADS) {
        const dfl z = df_from(zs[i]);
        dfl *t = ztab + ZTAB * i;
        t[0] = z;
        if (P.diag) {
            int b;
            t[2] = split_cell(df_mul(P.dic[8], z), b);
            t[1] = {__int_as_float(b), 0.f};
        } else {
#pragma unroll
            for (int k = 0; k < 3; k++) t[1 + k] = df_mul(P.dic[3 * k + 2], z);
        }
    }
    __syncthreads();
}

// TPS lanes per stroke (1, 2, 4 or 8): the lanes of a group hold the same state and split
// each trilinear gather (interp_force_df_group, bit-identical to one lane); lane 0 of the
// group writes the outputs.  More lanes per stroke put more warps in flight when a scan has
// few strokes, which is what bounds this kernel.  KEEP (one lane): the corner values of the
// stroke's cell are kept until it leaves it.
template <bool SCAN, int TPS, bool SPL, bool KEEP>
__global__ void __launch_bounds__(RELAX_THREADS) relax_kernel(const RelaxPrm P, const StrokeIO S, const ScanIO C) {
    extern __shared__ dfl ztab[];
    const int s = (blockIdx.x * RELAX_THREADS + threadIdx.x) / TPS;
    const int sub = (int)(threadIdx.x % TPS);
    const bool lead = sub == 0;
    const int nstroke = SCAN ? C.nx * C.ny : S.nstroke;
    const int nstep = SCAN ? C.nz : S.nstep;
    if (SCAN) fill_ztab(ztab, P, C.zs, nstep);
    bool active = s < nstroke && nstep > 0;

    int ix = 0, iy = 0;
    if (SCAN && active) {
        ix = s / C.ny;
        iy = s - ix * C.ny;
    }
    // tip (double-float) and its grid coordinate: base cell + fraction
    dfl tip[3], gxy[3];
    int base[3];
    dfl tf[3];
    auto set_height = [&](int iz) {
        dfl g[3];
        if (SCAN && P.diag) {
            tip[2] = ztab[ZTAB * iz];
            base[2] = __float_as_int(ztab[ZTAB * iz + 1].h);
            tf[2] = ztab[ZTAB * iz + 2];
            return;
        }
        if (SCAN) {
            tip[2] = ztab[ZTAB * iz];
#pragma unroll
            for (int k = 0; k < 3; k++) g[k] = df_add(gxy[k], ztab[ZTAB * iz + 1 + k]);
        } else {
            const double *t = S.rTips + ((long long)s * nstep + iz) * 3;
            tip[0] = df_from(t[0]);
            tip[1] = df_from(t[1]);
            tip[2] = df_from(t[2]);
            grid_of(P.dic, P.diag, tip, g);
        }
        tip_cell(g, base, tf);
    };

    dfl d[3] = {P.r0[0], P.r0[1], P.r0[2]};  // first start: r = tip + rPP0
    float3 v = make_float3(0.f, 0.f, 0.f);
    float dt = P.dtmaxf, acoef = P.acoef0f;
    int iz = 0, it = 0, itcount = 0;
    bool fin = P.maxIters <= 0;
    int itsum = 0;
    unsigned long long mine = 0;
    if (active) {
        if (SCAN) {
            tip[0] = df_from(C.xs[ix]);
            tip[1] = df_from(C.ys[iy]);
            const dfl r[3] = {tip[0], tip[1], {0.f, 0.f}};
            grid_of(P.dic, P.diag, r, gxy);
            tip_cell(gxy, base, tf);
        }
        set_height(0);
    }

    Corners corners;  // KEEP
    corners.cell = -1;
    unsigned am;
    while ((am = __ballot_sync(FULL, active)) != 0u) {
        if (!active) continue;
        dfl u[3], F[3];
        grid_coord_df(P.dic, P.diag, tf, d, u);
        if constexpr (KEEP) interp_force_df(P.FE, P.n0, P.n1, P.n2, base, u, F, corners);
        else interp_force_df_group<TPS>(P.FE, P.n0, P.n1, P.n2, base, u, F, sub, am);
        if (fin) {
            // outputs of height iz: position after the last move, grid force there
            dfl r[3];
#pragma unroll
            for (int k = 0; k < 3; k++) r[k] = df_add(tip[k], d[k]);
            if (!lead) {
            } else if (SCAN) {
                const long long o = (long long)s * nstep + (nstep - 1 - iz);
                if (C.fzs) C.fzs[o] = df_round(F[2]);
                if (C.ppos) {
                    C.ppos[3 * o + 0] = df_round(df_add(r[0], C.offd[0]));
                    C.ppos[3 * o + 1] = df_round(df_add(r[1], C.offd[1]));
                    C.ppos[3 * o + 2] = df_round(df_add(r[2], C.offd[2]));
                }
                if (C.iters) C.iters[o] = itcount;
            } else {
                const long long o = (long long)s * nstep + iz;
                S.rs[3 * o + 0] = df_to(r[0]);
                S.rs[3 * o + 1] = df_to(r[1]);
                S.rs[3 * o + 2] = df_to(r[2]);
                S.fs[3 * o + 0] = df_to(F[0]);
                S.fs[3 * o + 1] = df_to(F[1]);
                S.fs[3 * o + 2] = df_to(F[2]);
                if (S.iters) S.iters[o] = itcount;
            }
            itsum += itcount;
            iz++;
            if (iz == nstep) {
                active = false;
                if (!SCAN && S.itrsum && lead) S.itrsum[s] = itsum;
                if (SCAN && C.df && C.fzs && C.nw > 0 && lead) {
                    // np.convolve(fzs, W, 'valid') along ascending z (Fz2df, common.py:421-430)
                    const float *f = C.fzs + (long long)s * nstep;
                    const int nout = nstep - C.nw + 1;
                    float *out = C.df + (long long)s * nout;
                    for (int j = 0; j < nout; j++) {
                        float acc = 0.f;
                        for (int i = 0; i < C.nw; i++) acc = fmaf(f[j + i], C.W[C.nw - 1 - i], acc);
                        out[j] = acc;
                    }
                }
                continue;
            }
            // next height: warm start (relaxTipStroke, ProbeParticle.cpp:643-655)
            set_height(iz);
            if (P.probeStart == 0) {
                d[0] = P.r0[0];
                d[1] = P.r0[1];
                d[2] = P.r0[2];
            } else if (P.probeStart == -1) {  // the probe stays where it was: d = r_old - tip_new
#pragma unroll
                for (int k = 0; k < 3; k++) d[k] = df_add(r[k], df_neg(tip[k]));
            }  // probeStart == 1: d = r - r_tip carries over unchanged
            v = make_float3(0.f, 0.f, 0.f);
            dt = P.dtmaxf;
            acoef = P.acoef0f;
            it = 0;
            fin = P.maxIters <= 0;
            itcount = 0;
            continue;
        }
        const float3 f = pp_force_df<SPL>(P, F, d);
        const float ff = relax_move_df(P, f, d, v, dt, acoef);
        mine += lead ? 1 : 0;
        if (ff < P.convF2f) {
            itcount = it;
            fin = true;
        } else if (++it >= P.maxIters) {
            itcount = P.maxIters;
            fin = true;
        }
    }
    add_iterations(P.iter_total, mine);
}

// ------------------------------------------------- three lanes a stroke, one for each axis
//
// relax_kernel with the axes of a stroke on three lanes (ten strokes a warp): lane k holds the
// k-th component of the displacement, the velocity and the tip, computes the k-th grid coordinate,
// interpolates the k-th force component and moves along it; cell offsets, fractions, squares and
// dot products pass between the three by shuffles.  Every operation is one of relax_kernel's on the
// same operands, so the results are the same bit for bit.  A trip takes ~450 instructions instead
// of ~800, so a stroke -- the longest of which sets a small scan's time -- ends sooner; all strokes
// together take more of them (3 x 450), so scans that fill the GPU stay with one lane.  Cells with a
// diagonal metric; the harmonic radial spring.  Bound by a trip's dependent chain (~1300 cycles: the
// double-float interpolation, the springs, three rounds of shuffles) and, at 160^2, by issue.
//
// Relaxed scan + df of a 38-atom molecule, 30 heights, before (one lane, gathering every trip) and
// now: 32^2 strokes 1.27 -> 0.80 ms, 160^2 1.62 -> 1.37.  The line: one lane with the kept corners
// against three, 128^2 1.22 against 0.98 ms, 160^2 1.38 against 1.19, 192^2 1.46 against 1.56,
// 512^2 (40 heights) 6.8 against 8.6.
constexpr int AXIS_MAX_STROKES = 30000;  // ~5 warps on each of 608 schedulers

template <bool SCAN>
__global__ void __launch_bounds__(RELAX_THREADS) relax_axis_kernel(const RelaxPrm P, const StrokeIO S, const ScanIO C) {
    extern __shared__ dfl ztab[];
    const int warp = threadIdx.x >> 5;
    const AxisLane al = axis_lane(threadIdx.x & 31);
    const int k = al.k;
    const int nstroke = SCAN ? C.nx * C.ny : S.nstroke;
    const int nstep = SCAN ? C.nz : S.nstep;
    const dfl dic = k == 0 ? P.dic[0] : (k == 1 ? P.dic[4] : P.dic[8]);
    const dfl nr0 = k == 0 ? P.nr0[0] : (k == 1 ? P.nr0[1] : P.nr0[2]);
    const dfl kS = k == 0 ? P.kSf[0] : (k == 1 ? P.kSf[1] : P.kSf[2]);
    const dfl r0 = k == 0 ? P.r0[0] : (k == 1 ? P.r0[1] : P.r0[2]);
    const dfl off = !SCAN ? dfl{0.f, 0.f} : (k == 0 ? C.offd[0] : (k == 1 ? C.offd[1] : C.offd[2]));
    const int n = k == 0 ? P.n0 : (k == 1 ? P.n1 : P.n2);
    const int pitch = k == 0 ? P.n1 * P.n2 : (k == 1 ? P.n2 : 1);
    if (SCAN) fill_ztab(ztab, P, C.zs, nstep);
    const long long s = ((long long)blockIdx.x * (RELAX_THREADS / 32) + warp) * AXIS_STROKES + al.grp;
    bool active = !al.spare && s < nstroke && nstep > 0;
    const float *fe = reinterpret_cast<const float *>(P.FE) + k;

    dfl tip = {0.f, 0.f}, tf = {0.f, 0.f}, d = r0;
    int base = 0;
    auto set_height = [&](int iz) {
        if (SCAN) {
            if (k == 2) {
                tip = ztab[ZTAB * iz];
                base = __float_as_int(ztab[ZTAB * iz + 1].h);
                tf = ztab[ZTAB * iz + 2];
            }
        } else {
            tip = df_from(S.rTips[(s * nstep + iz) * 3 + k]);
            tf = split_cell(df_mul(dic, tip), base);
        }
    };
    if (active) {
        if (SCAN && k < 2) {
            const int ix = (int)(s / C.ny), iy = (int)(s - (long long)ix * C.ny);
            tip = df_from(k == 0 ? C.xs[ix] : C.ys[iy]);
            tf = split_cell(df_mul(dic, tip), base);
        }
        set_height(0);
    }
    float v = 0.f, dt = P.dtmaxf, acoef = P.acoef0f;
    int iz = 0, it = 0, itcount = 0, itsum = 0;
    bool fin = P.maxIters <= 0;
    unsigned long long mine = 0;
    float c[8];  // the corner values of the cell that the stroke is in (Corners)
    int cell = -1;
    auto from = [&](float x, int a) { return __shfl_sync(FULL, x, axis_source(al, a)); };
    auto from_df = [&](dfl x, int a) -> dfl { return {from(x.h, a), from(x.l, a)}; };

    while (__any_sync(FULL, active)) {
        // the grid force along this axis (interp_force_df); strokes that have ended repeat their last
        dfl F;
        {
            int ci;
            const dfl t = split_cell(df_add(tf, df_mul(dic, d)), ci);
            int i0 = ci + base;
            i0 += i0 < 0 ? n : 0;
            i0 -= i0 >= n ? n : 0;
            if ((unsigned)i0 >= (unsigned)n) i0 = wrap_index(i0, n);  // more than one cell away
            const int i1 = (i0 + 1 == n) ? 0 : i0 + 1;
            const int a0 = i0 * pitch, a1 = i1 * pitch;
            dfl tt[3], m[3];
            int o[3][2];
#pragma unroll
            for (int a = 0; a < 3; a++) {
                o[a][0] = __shfl_sync(FULL, a0, axis_source(al, a));
                o[a][1] = __shfl_sync(FULL, a1, axis_source(al, a));
                tt[a] = from_df(t, a);
                const dfl q = fast_two_sum(1.f, -tt[a].h);
                m[a] = {q.h, __fsub_rn(q.l, tt[a].l)};
            }
            const int at = axis_corner(o, 0);
            if (at != cell) {
                cell = at;
#pragma unroll
                for (int j = 0; j < 8; j++) c[j] = __ldg(fe + 4 * (long long)axis_corner(o, j));
            }
            const dfl wxy[4] = {df_mul(m[0], m[1]), df_mul(m[0], tt[1]), df_mul(tt[0], m[1]), df_mul(tt[0], tt[1])};
            dfl p[8];
#pragma unroll
            for (int j = 0; j < 8; j++) {
                const dfl w = df_mul(wxy[j >> 1], (j & 1) ? tt[2] : m[2]);
                p[j] = two_prod(w.h, c[j]);
                p[j].l = __fmaf_rn(w.l, c[j], p[j].l);
            }
            const dfl r = df_add_raw(df_add_raw(df_add_raw(p[0], p[1]), df_add_raw(p[2], p[3])),
                                     df_add_raw(df_add_raw(p[4], p[5]), df_add_raw(p[6], p[7])));
            F = two_sum(r.h, r.l);
        }
        // the springs (pp_force_df)
        float f;
        {
            const dfl q = df_sq(d);
            const dfl l2 = df_add(df_add(from_df(q, 0), from_df(q, 1)), from_df(q, 2));
            const float rs = rsqrt_approx(l2.h);
            const float L = __fmul_rn(l2.h, rs);
            const dfl LL = two_prod(L, L);
            const float res = __fadd_rn(__fsub_rn(__fsub_rn(l2.h, LL.h), LL.l), l2.l);
            const dfl l = fast_two_sum(L, __fmul_rn(res, __fmul_rn(0.5f, rs)));
            const dfl x = df_add(l, P.nl0);
            const float qh = __fmul_rn(x.h, rs);
            const dfl ql = two_prod(qh, l.h);
            const float rem = __fsub_rn(__fadd_rn(__fsub_rn(__fsub_rn(x.h, ql.h), ql.l), x.l), __fmul_rn(qh, l.l));
            const dfl sp = df_mul(P.kRadf, two_sum(qh, __fmul_rn(rem, rs)));
            const dfl b = two_prod(d.h, sp.h);
            const float bl = __fmaf_rn(d.l, sp.h, __fmaf_rn(d.h, sp.l, b.l));
            const dfl r = two_sum(d.h, nr0.h);
            const float rl = __fadd_rn(r.l, __fadd_rn(d.l, nr0.l));
            const dfl c = two_prod(r.h, kS.h);
            const float cl = __fmaf_rn(rl, kS.h, __fmaf_rn(r.h, kS.l, c.l));
            const dfl s1 = two_sum(F.h, b.h);
            const dfl s2 = two_sum(s1.h, c.h);
            f = __fadd_rn(s2.h, __fadd_rn(__fadd_rn(s1.l, s2.l), __fadd_rn(F.l, __fadd_rn(bl, cl))));
        }
        const float fx = from(f, 0), fy = from(f, 1), fz = from(f, 2);
        const float vx = from(v, 0), vy = from(v, 1), vz = from(v, 2);
        // one move (relax_move_df), with selects for its branches
        const bool upd = active && !fin, done = active && fin;
        {
            const float ff = __fmaf_rn(fz, fz, __fmaf_rn(fy, fy, __fmul_rn(fx, fx)));
            const float vv = __fmaf_rn(vz, vz, __fmaf_rn(vy, vy, __fmul_rn(vx, vx)));
            const float vf = __fmaf_rn(fz, vz, __fmaf_rn(fy, vy, __fmul_rn(fx, vx)));
            const bool fire = P.relaxAlg == 1, back = vf < 0.f;
            const float vf2 = __fmul_rn(vv, ff);
            const float cf = (vf2 > 1e-30f) ? __fmul_rn(__fmul_rn(acoef, vv), rsqrt_approx(vf2)) : 0.f;
            float nv = __fmul_rn(v, __fsub_rn(1.f, fire ? acoef : P.acoef0f));
            if (fire) nv = back ? 0.f : __fmaf_rn(f, cf, nv);
            const float ndt = !fire ? dt : (back ? __fmul_rn(dt, P.fdecf) : fminf(__fmul_rn(dt, P.fincf), P.dtmaxf));
            const float nac = !fire ? acoef : (back ? P.acoef0f : __fmul_rn(acoef, P.falphaf));
            const float h = fire ? ndt : P.dtmaxf;
            nv = __fmaf_rn(f, h, nv);
            const dfl nd = df_add_f(d, __fmul_rn(nv, h));
            const bool conv = ff < P.convF2f;
            const int nit = it + (conv ? 0 : 1);
            if (upd) {
                v = nv;
                dt = ndt;
                acoef = nac;
                mine += k == 0 ? 1 : 0;
                fin = conv || nit >= P.maxIters;
                it = nit;
                itcount = conv ? it : P.maxIters;
            }
            d.h = upd ? nd.h : d.h;
            d.l = upd ? nd.l : d.l;
        }
        if (done) {
            const dfl r = df_add(tip, d);
            if (SCAN) {
                const long long o = s * nstep + (nstep - 1 - iz);
                if (C.fzs && k == 2) C.fzs[o] = df_round(F);
                if (C.ppos) C.ppos[3 * o + k] = df_round(df_add(r, off));
                if (C.iters && k == 0) C.iters[o] = itcount;
            } else {
                const long long o = s * nstep + iz;
                S.rs[3 * o + k] = df_to(r);
                S.fs[3 * o + k] = df_to(F);
                if (S.iters && k == 0) S.iters[o] = itcount;
            }
            itsum += itcount;
            iz++;
            if (iz == nstep) {
                active = false;
                if (!SCAN && S.itrsum && k == 0) S.itrsum[s] = itsum;
                if (SCAN && C.df && C.fzs && C.nw > 0 && k == 2) {  // this lane wrote the stroke's fzs
                    const float *fr = C.fzs + s * nstep;
                    const int nout = nstep - C.nw + 1;
                    float *out = C.df + s * nout;
                    for (int j = 0; j < nout; j++) {
                        float acc = 0.f;
                        for (int i = 0; i < C.nw; i++) acc = fmaf(fr[j + i], C.W[C.nw - 1 - i], acc);
                        out[j] = acc;
                    }
                }
            } else {
                set_height(iz);
                if (P.probeStart == 0) d = r0;
                else if (P.probeStart == -1) d = df_add(r, df_neg(tip));
                v = 0.f;
                dt = P.dtmaxf;
                acoef = P.acoef0f;
                it = 0;
                fin = P.maxIters <= 0;
                itcount = 0;
            }
        }
    }
    add_iterations(P.iter_total, mine);
}

// ------------------------------------------------------------- AFMulator semantics

struct AfmPrm {
    const float4 *FE;
    int n0, n1, n2;
    float dic[9];  // rows: transpose(inv(cell)) row k times n_k
    float dtmax, damp0;
    float stiff[4], dpos0[4];
    float tA[3], tB[3], tC[3], zstep_w;
    float surf;
    int npix, nz;
    const float4 *points;
    float4 *FEs, *paths;
    int *iters;
    float *X;
    int nw;
    float W[MAX_DF_TAPS];
    unsigned long long *iter_total;
};

__device__ __forceinline__ float dot3(float3 a, const float *b) { return a.x * b[0] + a.y * b[1] + a.z * b[2]; }

constexpr int AFM_RELAX_THREADS = 128;  // as the single-grid kernel: packs beside the next image's force field

template <bool KEEP>
__global__ void __launch_bounds__(AFM_RELAX_THREADS) relax_afm_kernel(const AfmPrm P) {
    const int p = blockIdx.x * AFM_RELAX_THREADS + threadIdx.x;
    bool active = p < P.npix && P.nz > 0;
    const float3 dTip = make_float3(P.tC[0] * P.zstep_w, P.tC[1] * P.zstep_w, P.tC[2] * P.zstep_w);
    // dpos0 rotated to the lab frame (rotMatT)
    const float3 d0 = make_float3(P.tA[0] * P.dpos0[0] + P.tB[0] * P.dpos0[1] + P.tC[0] * P.dpos0[2],
                                  P.tA[1] * P.dpos0[0] + P.tB[1] * P.dpos0[1] + P.tC[1] * P.dpos0[2],
                                  P.tA[2] * P.dpos0[0] + P.tB[2] * P.dpos0[1] + P.tC[2] * P.dpos0[2]);
    float3 tip = make_float3(0.f, 0.f, 0.f), pos = tip;
    if (active) {
        const float4 q = P.points[p];
        tip = make_float3(q.x, q.y, q.z);
        pos = make_float3(tip.x + d0.x, tip.y + d0.y, tip.z + d0.z);
    }
    float dt = P.dtmax, damp = P.damp0;
    const float dtmin = P.dtmax * 0.1f;
    float3 v = make_float3(0.f, 0.f, 0.f);
    int iz = 0, it = 0;
    unsigned long long mine = 0;
    constexpr int NMAX = 128;  // N_RELAX_STEP_MAX (relax.cl:90)
    Corners4 corners;

    while (__any_sync(FULL, active)) {
        if (!active) continue;
        float3 g;
        g.x = dot3(pos, P.dic);
        g.y = dot3(pos, P.dic + 3);
        g.z = dot3(pos, P.dic + 6);
        const float4 fe = interp_fe4<KEEP>(P.FE, P.n0, P.n1, P.n2, g, corners);
        float3 f = make_float3(fe.x, fe.y, fe.z);
        const float3 dp = make_float3(pos.x - tip.x, pos.y - tip.y, pos.z - tip.z);
        const float3 dq = make_float3(dot3(dp, P.tA), dot3(dp, P.tB), dot3(dp, P.tC));
        const float r = sqrtf(dq.x * dq.x + dq.y * dq.y + dq.z * dq.z);
        const float rad = P.stiff[3] * (r - P.dpos0[3]) / r;
        const float3 ft = make_float3((dq.x - P.dpos0[0]) * P.stiff[0] + dq.x * rad,
                                      (dq.y - P.dpos0[1]) * P.stiff[1] + dq.y * rad,
                                      (dq.z - P.dpos0[2]) * P.stiff[2] + dq.z * rad);
        f.x += P.tA[0] * ft.x + P.tB[0] * ft.y + P.tC[0] * ft.z + P.tC[0] * P.surf;
        f.y += P.tA[1] * ft.x + P.tB[1] * ft.y + P.tC[1] * ft.z + P.tC[1] * P.surf;
        f.z += P.tA[2] * ft.x + P.tB[2] * ft.y + P.tC[2] * ft.z + P.tC[2] * P.surf;
        // update_FIRE (relax.cl:105-126)
        const float ff = f.x * f.x + f.y * f.y + f.z * f.z;
        const float vv = v.x * v.x + v.y * v.y + v.z * v.z;
        const float vf = v.x * f.x + v.y * f.y + v.z * f.z;
        if (vf < 0.f) {
            v = make_float3(0.f, 0.f, 0.f);
            dt = fmaxf(dtmin, dt * 0.5f);
            damp = P.damp0;
        } else {
            const float cf = damp * sqrtf(vv / (ff + 1e-8f));
            const float cv = 1.f - damp;
            v.x = fmaf(f.x, cf, v.x * cv);
            v.y = fmaf(f.y, cf, v.y * cv);
            v.z = fmaf(f.z, cf, v.z * cv);
            dt = fminf(P.dtmax, dt * 1.1f);
            damp *= 0.99f;
        }
        v.x = fmaf(f.x, dt, v.x);
        v.y = fmaf(f.y, dt, v.y);
        v.z = fmaf(f.z, dt, v.z);
        pos.x = fmaf(v.x, dt, pos.x);
        pos.y = fmaf(v.y, dt, pos.y);
        pos.z = fmaf(v.z, dt, pos.z);
        mine++;
        it++;
        if (ff < 1e-8f || it >= NMAX) {
            const long long o = (long long)p * P.nz + iz;
            if (P.FEs) {
                float4 r4;
                r4.x = fe.x * P.tA[0] + fe.y * P.tA[1] + fe.z * P.tA[2];
                r4.y = fe.x * P.tB[0] + fe.y * P.tB[1] + fe.z * P.tB[2];
                r4.z = fe.x * P.tC[0] + fe.y * P.tC[1] + fe.z * P.tC[2];
                r4.w = fe.w;
                P.FEs[o] = r4;
            }
            if (P.paths) P.paths[o] = make_float4(pos.x, pos.y, pos.z, 0.f);
            if (P.iters) P.iters[o] = (ff < 1e-8f) ? it - 1 : NMAX;
            tip.x += dTip.x;
            tip.y += dTip.y;
            tip.z += dTip.z;
            pos.x += dTip.x;
            pos.y += dTip.y;
            pos.z += dTip.z;
            v = make_float3(0.f, 0.f, 0.f);
            it = 0;
            iz++;
            if (iz == P.nz) {
                active = false;
                if (P.X && P.FEs && P.nw > 0) {
                    // convolveZ (relax.cl:571-608): X[o] = sum_j FEs[o+j].z * W[j]
                    const float4 *fin = P.FEs + (long long)p * P.nz;
                    const int nout = P.nz - P.nw + 1;
                    float *out = P.X + (long long)p * nout;
                    for (int o2 = 0; o2 < nout; o2++) {
                        float acc = 0.f;
                        for (int j = 0; j < P.nw; j++) acc = fmaf(fin[o2 + j].z, P.W[j], acc);
                        out[o2] = acc;
                    }
                }
            }
        }
    }
    add_iterations(P.iter_total, mine);
}

// relax_afm_kernel with a stroke on four lanes (eight strokes a warp): lanes 0-2 hold an axis each,
// as in relax_axis_kernel, lane 3 interpolates the energy; the branches of the FIRE step are
// selects.  The same operations on the same operands: the same results bit for bit.
//   128^2 strokes of 30 heights, one lane -> four: 0.785 -> 0.505 ms, 16^2 0.77 -> 0.46,
//   192^2 0.84 -> 0.75, 256^2 0.94 -> 1.16.  Bound by a trip's dependent chain (two square roots,
//   two divisions, an interpolation), one warp a scheduler.
constexpr int AFM_GROUP = 4;
constexpr int AFM_AXIS_MAX_STROKES = 40000;

__global__ void __launch_bounds__(AFM_RELAX_THREADS) relax_afm_axis_kernel(const AfmPrm P) {
    const int lane = threadIdx.x & 31, k = lane & 3, a = k < 3 ? k : 2;  // a: the axis of a lane's position
    const long long p = ((long long)blockIdx.x * AFM_RELAX_THREADS + threadIdx.x) / AFM_GROUP;
    bool active = p < P.npix && P.nz > 0;
    auto pick3 = [&](const float *v) { return a == 0 ? v[0] : (a == 1 ? v[1] : v[2]); };
    const float tAk = pick3(P.tA), tBk = pick3(P.tB), tCk = pick3(P.tC);
    const float dic[3] = {a == 0 ? P.dic[0] : (a == 1 ? P.dic[3] : P.dic[6]), a == 0 ? P.dic[1] : (a == 1 ? P.dic[4] : P.dic[7]),
                          a == 0 ? P.dic[2] : (a == 1 ? P.dic[5] : P.dic[8])};
    const int n = a == 0 ? P.n0 : (a == 1 ? P.n1 : P.n2), pitch = a == 0 ? P.n1 * P.n2 : (a == 1 ? P.n2 : 1);
    const float *fep = reinterpret_cast<const float *>(P.FE) + k;
    const float dTip = tCk * P.zstep_w;
    float tip = 0.f, pos = 0.f;
    if (active) {
        const float4 q = P.points[p];
        tip = a == 0 ? q.x : (a == 1 ? q.y : q.z);
        pos = tip + (tAk * P.dpos0[0] + tBk * P.dpos0[1] + tCk * P.dpos0[2]);
    }
    float dt = P.dtmax, damp = P.damp0, v = 0.f;
    const float dtmin = P.dtmax * 0.1f;
    int iz = 0, it = 0, cell = -1;
    float c[8] = {};
    unsigned long long mine = 0;
    constexpr int NMAX = 128;  // N_RELAX_STEP_MAX (relax.cl:90)
    auto from = [&](float x, int l) { return __shfl_sync(FULL, x, l, AFM_GROUP); };

    while (__any_sync(FULL, active)) {
        const float px = from(pos, 0), py = from(pos, 1), pz = from(pos, 2);
        const float g = px * dic[0] + py * dic[1] + pz * dic[2];
        const float fl = floorf(g), t = g - fl;
        int i0 = (int)fl;
        i0 += i0 < 0 ? n : 0;
        i0 -= i0 >= n ? n : 0;
        if ((unsigned)i0 >= (unsigned)n) i0 = wrap_index(i0, n);
        const int i1 = (i0 + 1 == n) ? 0 : i0 + 1;
        const int a0 = i0 * pitch, a1 = i1 * pitch;
        int o[3][2];
#pragma unroll
        for (int l = 0; l < 3; l++) {
            o[l][0] = __shfl_sync(FULL, a0, l, AFM_GROUP);
            o[l][1] = __shfl_sync(FULL, a1, l, AFM_GROUP);
        }
        const float tx = from(t, 0), ty = from(t, 1), tz = from(t, 2);
        const float mx = 1.f - tx, my = 1.f - ty, mz = 1.f - tz;
        const int at = o[0][0] + o[1][0] + o[2][0];
        if (at != cell) {
            cell = at;
#pragma unroll
            for (int j = 0; j < 8; j++) c[j] = __ldg(fep + 4 * (long long)(o[0][j >> 2] + o[1][(j >> 1) & 1] + o[2][j & 1]));
        }
        const float v00 = fmaf(c[4], tx, c[0] * mx), v10 = fmaf(c[6], tx, c[2] * mx);
        const float v01 = fmaf(c[5], tx, c[1] * mx), v11 = fmaf(c[7], tx, c[3] * mx);
        const float v0 = fmaf(v10, ty, v00 * my), v1 = fmaf(v11, ty, v01 * my);
        const float fe = fmaf(v1, tz, v0 * mz);
        const float dpk = pos - tip;
        const float3 dp = make_float3(from(dpk, 0), from(dpk, 1), from(dpk, 2));
        const float3 dq = make_float3(dot3(dp, P.tA), dot3(dp, P.tB), dot3(dp, P.tC));
        const float r = sqrtf(dq.x * dq.x + dq.y * dq.y + dq.z * dq.z);
        const float rad = P.stiff[3] * (r - P.dpos0[3]) / r;
        const float3 ft = make_float3((dq.x - P.dpos0[0]) * P.stiff[0] + dq.x * rad,
                                      (dq.y - P.dpos0[1]) * P.stiff[1] + dq.y * rad,
                                      (dq.z - P.dpos0[2]) * P.stiff[2] + dq.z * rad);
        float fk = fe;
        fk += tAk * ft.x + tBk * ft.y + tCk * ft.z + tCk * P.surf;
        const float3 f = make_float3(from(fk, 0), from(fk, 1), from(fk, 2));
        const float3 w = make_float3(from(v, 0), from(v, 1), from(v, 2));
        // update_FIRE (relax.cl:105-126)
        const float ff = f.x * f.x + f.y * f.y + f.z * f.z;
        const float vv = w.x * w.x + w.y * w.y + w.z * w.z;
        const float vf = w.x * f.x + w.y * f.y + w.z * f.z;
        const bool back = vf < 0.f;
        const float cf = damp * sqrtf(vv / (ff + 1e-8f));
        const float cv = 1.f - damp;
        const float nv = back ? 0.f : fmaf(fk, cf, v * cv);
        const float nd = back ? fmaxf(dtmin, dt * 0.5f) : fminf(P.dtmax, dt * 1.1f);
        if (active) {
            damp = back ? P.damp0 : damp * 0.99f;
            dt = nd;
            v = fmaf(fk, nd, nv);
            pos = fmaf(v, nd, pos);
            mine += k == 0 ? 1 : 0;
            it++;
        }
        const bool end = active && (ff < 1e-8f || it >= NMAX);
        if (__any_sync(FULL, end)) {
            const float3 q = make_float3(from(fe, 0), from(fe, 1), from(fe, 2));
            if (end) {
                const long long o4 = p * P.nz + iz;
                // lanes 0-2: the force along A, B, C; lane 3: the energy
                const float *row = k == 0 ? P.tA : (k == 1 ? P.tB : P.tC);
                const float rec = q.x * row[0] + q.y * row[1] + q.z * row[2];
                if (P.FEs) reinterpret_cast<float *>(P.FEs + o4)[k] = k < 3 ? rec : fe;
                if (P.paths) reinterpret_cast<float *>(P.paths + o4)[k] = k < 3 ? pos : 0.f;
                if (P.iters && k == 0) P.iters[o4] = (ff < 1e-8f) ? it - 1 : NMAX;
                tip += dTip;
                pos += dTip;
                v = 0.f;
                it = 0;
                iz++;
                if (iz == P.nz) {
                    active = false;
                    if (P.X && P.FEs && P.nw > 0 && k == 2) {  // this lane wrote the stroke's FEs.z
                        const float4 *fin = P.FEs + p * P.nz;
                        const int nout = P.nz - P.nw + 1;
                        float *out = P.X + p * nout;
                        for (int o2 = 0; o2 < nout; o2++) {
                            float acc = 0.f;
                            for (int j = 0; j < P.nw; j++) acc = fmaf(fin[o2 + j].z, P.W[j], acc);
                            out[o2] = acc;
                        }
                    }
                }
            }
        }
    }
    add_iterations(P.iter_total, mine);
}

// ---------------------------------------------------------------------- host

TipSpline g_tip_spline = {0, nullptr, nullptr};
static void *g_spline_mem = nullptr;
static std::vector<double> g_spline_xs, g_spline_ydys;  // host copies (for save/restore)

// Uploads the spline tables (see TipSpline); n == 0 clears.  cudaFree of the previous tables
// waits for the kernels that may still read them.
static int upload_tip_spline(int n, const double *xs, const double *ydys) {
    if (n == 0 || !xs || !ydys) {
        if (g_spline_mem) cudaFree(g_spline_mem);
        g_spline_mem = nullptr;
        g_tip_spline = {0, nullptr, nullptr};
        g_spline_xs.clear();
        g_spline_ydys.clear();
        return set_ok();
    }
    if (n < 2) return set_error(PPGPU_ERR_ARG, "tip spline: %d knots (at least 2)", n);
    std::vector<dfl> tab((size_t)n + 6 * (size_t)(n - 1));
    for (int i = 0; i < n; i++) tab[i] = df_from(xs[i]);
    for (int i = 0; i < n - 1; i++) {
        const double x0 = xs[i], dx = xs[i + 1] - x0, denom = 1 / dx;
        const double y0 = ydys[2 * i], y1 = ydys[2 * i + 2], dy0 = ydys[2 * i + 1] * dx, dy1 = ydys[2 * i + 3] * dx;
        const double y01 = y0 - y1;
        const double c[6] = {x0, denom, y0, dy0, -3 * y01 - 2 * dy0 - dy1, 2 * y01 + dy0 + dy1};
        for (int k = 0; k < 6; k++) tab[n + 6 * i + k] = df_from(c[k]);
    }
    void *mem = nullptr;
    cudaError_t e = cudaMalloc(&mem, tab.size() * sizeof(dfl));
    if (e != cudaSuccess) return cuda_fail(e, "tip spline tables");
    e = cudaMemcpy(mem, tab.data(), tab.size() * sizeof(dfl), cudaMemcpyHostToDevice);
    if (e != cudaSuccess) {
        cudaFree(mem);
        return cuda_fail(e, "tip spline upload");
    }
    if (g_spline_mem) cudaFree(g_spline_mem);
    g_spline_mem = mem;
    g_tip_spline = {n, (const dfl *)mem, (const dfl *)mem + n};
    g_spline_xs.assign(xs, xs + n);
    g_spline_ydys.assign(ydys, ydys + 2 * (size_t)n);
    return set_ok();
}

// Runs fn with the tip spline (n, xs, ydys) in place of the current one, then restores it.
int with_tip_spline(int n, const double *xs, const double *ydys, int (*fn)(void *), void *arg) {
    std::vector<double> sx = g_spline_xs, sy = g_spline_ydys;
    const int n0 = (int)sx.size();
    int s = upload_tip_spline(n, xs, ydys);
    if (s) return s;
    s = fn(arg);
    const std::string msg = s ? std::string(ppgpu_last_error()) : std::string();
    const int st = s ? ppgpu_last_status() : 0;
    const int r = upload_tip_spline(n0, n0 ? sx.data() : nullptr, n0 ? sy.data() : nullptr);
    if (s) return set_error(st, "%s", msg.c_str());
    return r;
}

// Lanes per stroke that share its gathers (ppgpu_set_relax_tps).  One is the default: the scans
// measured here (16k-26k strokes) ran 15-20 % slower with 4, because every lane of a group also
// executes the stroke's FIRE arithmetic, which outweighs the latency hidden by the extra warps.
static int g_relax_tps = 0;  // 0: the default

static int relax_tps(long long) { return g_relax_tps ? g_relax_tps : 1; }

// Strokes keep the corners of their cell (Corners, Corners4) while all of them fit the GPU at once: the
// registers cost a CTA a SM (122 instead of 96: 4 instead of 5; the AFMulator's 79 instead of 56: 6
// instead of 9), which a scan of one wave does not miss and a larger one does.  One lane, 30 heights, every trip
// gathered against corners kept, ms: 180^2 strokes 1.21, 1.17, 260^2 (67 600) 1.82, 1.78, but 300^2 2.24, 2.36, 420^2 4.09, 4.14; with a
// tip spline 260^2 2.30, 2.26, 300^2 2.78, 3.17, 512^2 7.13, 7.47; on a tilted cell 260^2 2.04, 2.02, 300^2 2.50, 2.63.
// AFMulator: 256^2 1.01, 0.94, 340^2 (115 600) 1.25, 1.17, 400^2 1.61, 1.63, 640^2 3.27, 3.38.
constexpr long long KEEP_MAX_STROKES = 4LL * 152 * RELAX_THREADS;
constexpr long long AFM_KEEP_MAX_STROKES = 6LL * 152 * AFM_RELAX_THREADS;

template <bool SCAN, bool SPL>
static void launch_relax_t(int tps, bool keep, unsigned nblk, size_t smem, cudaStream_t st, const RelaxPrm &P, const StrokeIO &S,
                           const ScanIO &C) {
    switch (tps) {
    case 8: relax_kernel<SCAN, 8, SPL, false><<<nblk, RELAX_THREADS, smem, st>>>(P, S, C); break;
    case 4: relax_kernel<SCAN, 4, SPL, false><<<nblk, RELAX_THREADS, smem, st>>>(P, S, C); break;
    case 2: relax_kernel<SCAN, 2, SPL, false><<<nblk, RELAX_THREADS, smem, st>>>(P, S, C); break;
    default:
        if (keep) relax_kernel<SCAN, 1, SPL, true><<<nblk, RELAX_THREADS, smem, st>>>(P, S, C);
        else relax_kernel<SCAN, 1, SPL, false><<<nblk, RELAX_THREADS, smem, st>>>(P, S, C);
    }
}

template <bool SCAN>
static void launch_relax(int tps, long long nstroke, size_t smem, cudaStream_t st, const RelaxPrm &P, const StrokeIO &S,
                         const ScanIO &C) {
    if (g_relax_tps == 0 && nstroke <= AXIS_MAX_STROKES && P.diag && P.spl.n == 0 && (long long)P.n0 * P.n1 * P.n2 <= 0x7fffffffLL) {
        const long long warps = (nstroke + AXIS_STROKES - 1) / AXIS_STROKES;
        const unsigned nblk = (unsigned)((warps + RELAX_THREADS / 32 - 1) / (RELAX_THREADS / 32));
        relax_axis_kernel<SCAN><<<nblk, RELAX_THREADS, smem, st>>>(P, S, C);
        return;
    }
    const unsigned nblk = (unsigned)((nstroke * tps + RELAX_THREADS - 1) / RELAX_THREADS);
    const bool keep = nstroke <= KEEP_MAX_STROKES;
    if (P.spl.n > 0)
        launch_relax_t<SCAN, true>(tps, keep, nblk, smem, st, P, S, C);
    else
        launch_relax_t<SCAN, false>(tps, keep, nblk, smem, st, P, S, C);
}

}  // namespace ppgpu

using namespace ppgpu;

extern "C" int ppgpu_set_relax_tps(int tps) {
    if (tps != 0 && tps != 1 && tps != 2 && tps != 4 && tps != 8)
        return set_error(PPGPU_ERR_ARG, "set_relax_tps: %d not in {0 (default), 1, 2, 4, 8}", tps);
    g_relax_tps = tps;
    return set_ok();
}

extern "C" int ppgpu_set_tip_spline(int n, const double *xs, const double *ydys) {
    if (n < 0) return set_error(PPGPU_ERR_ARG, "set_tip_spline: negative knot count");
    return upload_tip_spline(n, xs, ydys);
}

extern "C" int ppgpu_get_relax_tps(long long nstroke, int *out) {
    if (!out || nstroke < 0) return set_error(PPGPU_ERR_ARG, "get_relax_tps: bad arguments");
    *out = relax_tps(nstroke);
    return set_ok();
}

extern "C" int ppgpu_relax_strokes(const float *FE, const int *n, const double *cell, const double *prm,
                                   int probeStart, int relaxAlg, int nstroke, int nstep, const double *rTips,
                                   double *rs, double *fs, int *iters, int *itrsum,
                                   unsigned long long *iter_total, void *stream) {
    if (!FE || !n || !cell || !prm) return set_error(PPGPU_ERR_ARG, "relax_strokes: null argument");
    if (nstroke < 0 || nstep < 0) return set_error(PPGPU_ERR_ARG, "relax_strokes: negative sizes");
    if (nstroke == 0 || nstep == 0) return set_ok();
    if (!rTips || !rs || !fs) return set_error(PPGPU_ERR_ARG, "relax_strokes: null stroke arrays");
    RelaxPrm P;
    int st = fill_relax_prm(P, FE, n, cell, prm, probeStart, relaxAlg, iter_total);
    if (st) return st;
    StrokeIO S = {nstroke, nstep, rTips, rs, fs, iters, itrsum};
    ScanIO C;
    memset(&C, 0, sizeof(C));
    launch_relax<false>(relax_tps(nstroke), nstroke, 0, (cudaStream_t)stream, P, S, C);
    PPGPU_CHECK_LAUNCH("relax_kernel<strokes>");
    return set_ok();
}

extern "C" int ppgpu_relax_scan(const float *FE, const int *n, const double *cell, const double *prm, int nx, int ny,
                                int nz, const double *xs, const double *ys, const double *zs,
                                const double *pos_offset, float *fzs, float *ppos, int *iters, int nw,
                                const double *df_weights, float *df, unsigned long long *iter_total,
                                void *stream) {
    if (!FE || !n || !cell || !prm || !xs || !ys || !zs) return set_error(PPGPU_ERR_ARG, "relax_scan: null argument");
    if (nx < 0 || ny < 0 || nz < 0) return set_error(PPGPU_ERR_ARG, "relax_scan: negative sizes");
    if (df && (nw <= 0 || nw > MAX_DF_TAPS || nw > nz || !df_weights || !fzs))
        return set_error(PPGPU_ERR_ARG, "relax_scan: df needs 1 <= nw <= min(64, nz), weights and fzs");
    if (nx == 0 || ny == 0 || nz == 0) return set_ok();
    RelaxPrm P;
    int st = fill_relax_prm(P, FE, n, cell, prm, 1, 1, iter_total);
    if (st) return st;
    StrokeIO S;
    memset(&S, 0, sizeof(S));
    ScanIO C;
    memset(&C, 0, sizeof(C));
    C.nx = nx;
    C.ny = ny;
    C.nz = nz;
    C.xs = xs;
    C.ys = ys;
    C.zs = zs;
    for (int k = 0; k < 3; k++) {
        C.off[k] = pos_offset ? pos_offset[k] : 0.0;
        C.offd[k] = df_from(C.off[k]);
    }
    C.fzs = fzs;
    C.ppos = ppos;
    C.iters = iters;
    C.df = df;
    C.nw = df ? nw : 0;
    for (int i = 0; i < C.nw; i++) C.W[i] = (float)df_weights[i];
    const long long npix = (long long)nx * ny;
    const size_t smem = (size_t)nz * ZTAB * sizeof(dfl);
    if (smem > 48 * 1024) return set_error(PPGPU_ERR_ARG, "relax_scan: nz = %d heights exceed the table limit (1536)", nz);
    launch_relax<true>(relax_tps(npix), npix, smem, (cudaStream_t)stream, P, S, C);
    PPGPU_CHECK_LAUNCH("relax_kernel<scan>");
    return set_ok();
}

extern "C" int ppgpu_relax_afm(const float *FE, const int *n, const double *inv_cell, const double *prm, int npix,
                               const float *points, int nz, float *FEs, float *paths, int *iters, int nw,
                               const double *weights, float *X, unsigned long long *iter_total, void *stream) {
    if (!FE || !n || !inv_cell || !prm || (npix > 0 && !points))
        return set_error(PPGPU_ERR_ARG, "relax_afm: null argument");
    if (X && (nw <= 0 || nw > MAX_DF_TAPS || nw > nz || !weights || !FEs))
        return set_error(PPGPU_ERR_ARG, "relax_afm: X needs 1 <= nw <= min(64, nz), weights and FEs");
    if (npix <= 0 || nz <= 0) return set_ok();
    AfmPrm P;
    memset(&P, 0, sizeof(P));
    P.FE = reinterpret_cast<const float4 *>(FE);
    P.n0 = n[0];
    P.n1 = n[1];
    P.n2 = n[2];
    for (int r = 0; r < 3; r++)
        for (int c = 0; c < 3; c++) P.dic[3 * r + c] = (float)(inv_cell[3 * r + c] * n[r]);
    P.dtmax = (float)prm[0];
    P.damp0 = (float)prm[1];
    for (int k = 0; k < 4; k++) {
        P.stiff[k] = (float)prm[4 + k];
        P.dpos0[k] = (float)prm[8 + k];
    }
    for (int k = 0; k < 3; k++) {
        P.tA[k] = (float)prm[12 + k];
        P.tB[k] = (float)prm[16 + k];
        P.tC[k] = (float)prm[20 + k];
    }
    P.zstep_w = (float)prm[23];
    P.surf = (float)prm[24];
    P.npix = npix;
    P.nz = nz;
    P.points = reinterpret_cast<const float4 *>(points);
    P.FEs = reinterpret_cast<float4 *>(FEs);
    P.paths = reinterpret_cast<float4 *>(paths);
    P.iters = iters;
    P.X = X;
    P.nw = X ? nw : 0;
    for (int i = 0; i < P.nw; i++) P.W[i] = (float)weights[i];
    P.iter_total = iter_total;
    if (npix <= AFM_AXIS_MAX_STROKES && (long long)P.n0 * P.n1 * P.n2 <= 0x7fffffffLL) {
        const unsigned nb = (unsigned)(((long long)npix * AFM_GROUP + AFM_RELAX_THREADS - 1) / AFM_RELAX_THREADS);
        relax_afm_axis_kernel<<<nb, AFM_RELAX_THREADS, 0, (cudaStream_t)stream>>>(P);
        PPGPU_CHECK_LAUNCH("relax_afm_axis_kernel");
        return set_ok();
    }
    const unsigned nblk = (unsigned)((npix + AFM_RELAX_THREADS - 1) / AFM_RELAX_THREADS);
    if (npix <= AFM_KEEP_MAX_STROKES) relax_afm_kernel<true><<<nblk, AFM_RELAX_THREADS, 0, (cudaStream_t)stream>>>(P);
    else relax_afm_kernel<false><<<nblk, AFM_RELAX_THREADS, 0, (cudaStream_t)stream>>>(P);
    PPGPU_CHECK_LAUNCH("relax_afm_kernel");
    return set_ok();
}
