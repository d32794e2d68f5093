// pp_ff_box.cu -- which force-field grids are summed by boxes (pp_ff_box_kern.cuh), and with how many
// nodes and levels; the kernels with 8 nodes (pp_ff_box10.cu has those with 10).
#include "pp_ff_box_kern.cuh"

namespace ppgpu {

// kappa: the interpolation error is 1.5e-7 of the r^-7 force, or 1.5e-8 of the Coulomb force alone.
static double box_kappa(int N, int mode) { return mode == M_COUL ? (N == 8 ? 4.5 : 3.0) : (N == 8 ? 7.0 : 4.25); }

// Largest distance of a tip charge from the probe's position.
static double tip_reach(const FFParams &prm) {
    double q = 0.0;
    for (int k = 0; k < prm.nqa; k++) q = std::max(q, (double)fabsf(prm.QZa[k]));
    return q;
}

// Grids and atoms summed by boxes.  Measured on a GB300, ff_block -> boxes (LJ + Coulomb, all atoms
// charged, 0.05 to 0.3 A steps alike):
//   200^3 points,   342 atoms          1.39 -> 0.28 ms     400x400x250, 18540 atoms  270 -> 5.8 ms,
//                                                          800x800x500                2120 -> 16.2 ms
//   128^3 (512 leaves): 540 atoms      0.61 -> 0.19 ms,  90: 0.113 -> 0.060,  60: 0.083 -> 0.077, 20: 0.041 -> 0.050
//   220^3 (2744 leaves): 90 atoms      0.51 -> 0.20 ms,  60: 0.36 -> 0.22,    20: 0.15 -> 0.165
//   96^3 (216 leaves): 540 atoms       0.28 -> 0.16 ms,  270: 0.146 -> 0.108;   80^3 (125), 1500: 0.49 -> 0.18
//   64^3 (64 leaves):  1500 atoms      0.30 -> 0.20 ms,  540: 0.108 -> 0.152, too few boxes to fill 152 SMs
//   AFMulator tip, 256x256x192:        38 atoms 1.05 -> 0.48 ms, 10 atoms 0.33 -> 0.23
// A box costs some 10 pairs a point whatever its atoms (classifying, interpolating, writing), which
// the far atoms have to save (more with fewer boxes than fill two CTAs a SM: tilted grids with energies of
// 68x34x239 points, 261 atoms 0.135 -> 0.32 ms); a pair with the tip's charges counts for five.  Where kappa H passes
// 36 A nearly every atom is near, and past 24 A in a solid more than the lists hold (slab on 64x64x40: 2.3
// -> 3.8 ms), which few boxes do not make up for.
//   Nodes: 10 leave a third of the near atoms at twice the work for a far one and for the levels,
// which pays from about 0.45 atoms a leaf (8 -> 10 nodes): 400x400x250, 18540 atoms (1.9 a leaf) 7.8 ->
// 5.7 ms, 240x240x150 (8) 9.0 -> 4.0, 128^3, 540 (1.05) 0.216 -> 0.193, 160^3, 540 (0.54) 0.253 -> 0.229, but
// 260^3, 1500 (0.3) 0.63 -> 0.72, 200^3, 342 (0.16) 0.28 -> 0.35.  The level above the leaves that 10 nodes need costs
// some 40 us (127x54x186, 216 atoms 0.138 without it -> 0.174), which few atoms pay only at coarse steps, where 7 H
// reaches most of them (112x52x123 at 0.215 A, 378 atoms 0.23 -> 0.16).  The 8 sums of LJ + Coulomb with the energy do not
// fit the registers as well (79x251x147, 459 atoms 0.34 -> 0.44, without the energy 0.30 -> 0.27).
//   Levels above the leaves, with 8 nodes: 220^3, 342 atoms 0.45, 0.31, 0.34 ms with 0, 1, 2 (9.4e5
// atom-boxes), 128^3, 540 atoms 0.216, 0.224 (2.8e5), 79x251x147, 459 0.335, 0.300 (3.7e5), 320^3, 540 atoms 1.70, 0.79, 0.73 (4.3e6); with 10
// nodes and 1, 2, 3: 128^3, 540 atoms 0.193, 0.214, 0.232 (2.8e5), slab on 240x240x150 6.6, 4.0, 4.1 (4.2e7), on
// 320x320x200 11.6, 5.07, 4.95 (9.3e7), on 400x400x250 18.8, 6.8, 5.7 (1.9e8).
//   Flat and narrow grids: a leaf of few points has no fewer nodes, and nothing can be handed to it that its
// points have no room for.  1x2000x2000 points, 342 atoms 0.70 against 2.66 ms by boxes, 1x1x20000, 1500 atoms 0.12 against 2.4,
// 4x400x400, 342 atoms 0.149 against 0.294 with 10 nodes (leaves of 1024 points, 1500 wanted), but 6x400x400, 18540 atoms (LJ)
// 7.4 against 0.87, 8x200x200, 1500 atoms 0.36 against 0.21.  So the sums have to fit a leaf (10 nodes pay from 1800 points,
// 8 without anything handed down from 1024), and leaves below 2000 points take as many more atoms.
//   Few boxes whose reach is long: nearly all atoms are near ones, unless they fill much more space than that.  51x32x136 points at
// 0.34 A, solid of 3869 atoms 0.58 against 1.38 ms, 55x144x27 at 0.4 A, slab of 1967 0.30 against 0.55; but 18540 atoms of
// the slab on 101x101x63 at 0.4 A 5.5 against 2.8.  Below 240 boxes and beyond 14 A: atoms as many as the reach cubed.
//   10 nodes for their shorter reach alone: 23x188x258 at 0.47 A, 63 atoms 0.093 against 0.136, 22x15x2322 at 0.4 A, 234 atoms
// 0.095 against 0.192, 192x194x178 at 0.47, 297 atoms 1.05 against 0.28: half as many atoms again.
//   Of 3370 calls of plausible molecules, layers, slabs and solids (16 to 300 points an axis, half of them flat or narrow, 0.05 to 0.6
// A) 39 are slower by boxes than pair by pair, by 1.2 times in the mean.
struct BoxChoice {
    int N, levels;
    bool boxes;
};
static BoxChoice box_choice(const FFParams &prm, int mode, bool with_e, BoxPrm *B) {
    const double nat = mode == M_COUL ? prm.ncharged : prm.natoms, boxes = box_count(prm), work = nat * boxes;
    const double pairs = nat + (mode == M_QZS && prm.nqa > 0 ? 4.0 * prm.ncharged : 0.0);
    double need = 40.0 + (boxes >= 304 ? 20480.0 : (boxes >= 200 ? 51200.0 : 70000.0)) / boxes;
    BoxChoice c = {8, 0, false};
    if (!(boxes >= 64 && pairs >= need)) return c;  // small calls: planning takes a third of a microsecond
    const double reach = tip_reach(prm);
    const int NC = (with_e ? 4 : 3) * (mode == M_LJC ? 2 : 1);  // sums of a node
    double H;
    box_plan(prm, 8, box_kappa(8, mode), reach, B, &H);
    const double far8 = H * box_kappa(8, mode);
    const bool dense = mode == M_LJC && with_e ? nat >= 2.0 * boxes : nat >= 1.2 * boxes || (nat >= 0.45 * boxes && (work >= 1.1e5 || far8 >= 12.0));
    if (!prm.accumulate && (dense || far8 > 36.0)) {
        box_plan(prm, 10, box_kappa(10, mode), reach, B, &H);
        if (box_leaf(*B) >= std::max(1800, 250 * NC)) c.N = 10;
        else box_plan(prm, 8, box_kappa(8, mode), reach, B, &H);
    }
    if (c.N == 8) c.levels = work < 3e5 ? 0 : (work < 3e6 ? 1 : (work < 1e9 ? 2 : 3));
    else c.levels = work < 8e6 ? 1 : (work < 8e7 ? 2 : 3);
    B->levels = prm.accumulate ? 0 : c.levels;
    const double far = H * box_kappa(c.N, mode), leaf = box_leaf(*B);
    if (leaf < 2000.0) need *= 2000.0 / leaf;
    if (c.N == 10 && !dense) need *= 1.5;
    c.boxes = pairs >= need && far <= (boxes >= 304 ? 36.0 : 24.0);
    if (c.N == 8 && leaf < (B->levels == 0 ? 1024 : 128 * NC)) c.boxes = false;
    if (boxes < 240 && far > 14.0 && pairs < far * far * far) c.boxes = false;
    return c;
}

FFRoute ff_box_route(const FFParams &prm, int mode, bool with_e) {
    BoxPrm B;
    const BoxChoice c = box_choice(prm, mode, with_e, &B);
    return c.boxes ? FFRoute{c.N, B.levels} : FFRoute{0, 0};
}

bool launch_ff_box(const FFParams &prm, int mode, bool with_e, bool ortho, cudaStream_t st, int *rc) {
    BoxPrm B;
    const BoxChoice c = box_choice(prm, mode, with_e, &B);
    if (!c.boxes) return false;
    *rc = c.N == 8 ? launch_box_nodes<8>(prm, B, mode, with_e, ortho, st) : launch_ff_box10(prm, B, mode, with_e, ortho, st);
    return true;
}

}  // namespace ppgpu
