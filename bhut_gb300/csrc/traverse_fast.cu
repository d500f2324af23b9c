// Barnes-Hut traversal, form "fast": FP64-accurate results from float-float
// arithmetic on the FP32 pipe.
//
// On GB300 the FP64 pipe runs at about 1/70 of the FP32 pipe, and f32<->f64
// conversions at the FP64 rate, so the FP64 pair loop of k_traverse_exact is
// bound at ~1 TFLOP/s.  This kernel keeps every pair term to ~2^-44 relative
// (the sum of ~5e4 such terms is far inside the 1e-10 relative-L2 contract)
// while issuing only FP32 instructions in the hot loop:
//
//  * Coordinates are shifted to the tree's box centre and scaled by a power
//    of two into [-1/2, 1/2]; each coordinate is stored as hi + lo with hi on
//    the 2^-23 grid and lo the rest in FP32 (|lo| <= 2^-24), so hi_j - hi_i
//    is exact in FP32 and the displacement is known to about 2^-48.  Masses
//    are scaled by a power of two into [-1, 1] and split hi + lo.  Scales are
//    undone in FP64.
//  * r^2 + eps^2 is summed error-free; (r^2)^(-3/2) is the hardware rsqrt
//    refined by one correction step from the exactly computed residual
//    (Newton-Raphson for the inverse square root; carried to second order
//    in the checked term); m * w * dx and the accumulation are float-float
//    (Dekker/Knuth two-product and TwoSum, or sums biased by a leaf's bounds:
//    pair terms and figures in fast.cuh).
//  * A pair's relative error is dominated by the coordinates: about
//    2^-48 / sqrt(r^2 + eps^2).  With a softening that bounds r^2 + eps^2
//    from below ((eps s)^2 >= 2^-33) every pair is float-float and the range
//    test is compiled out; otherwise pairs with r^2 + eps^2 below 2^-26 in
//    normalised units (softened distance under 2^-13 of the box half-size),
//    or outside the FP32 range, are evaluated in FP64 from the FP64 arrays,
//    so a float-float pair stays below 2^-35.
//  * The opening decision is the reference's, bit for bit: a FP32 test
//    decides every node whose ratio is clearly above or below theta, and
//    nodes inside a small error band are decided by the exact FP64 test of
//    k_traverse_exact (bh.py:576-601).  Every lane therefore evaluates
//    exactly the reference's interaction set for its target.
#include <cmath>

#include "fast.cuh"

namespace bhut {

constexpr int kFastWarps = 4;
constexpr int kFastThreads = kFastWarps * kWarp;
// Tuning (overridable at build time): resident blocks per SM of the fast form
// (they cap the registers: 5 / 6 / 7 / 8 at 96 / 80 / 72 / 64).
//   3-D, softened, not split: 5 / 6 / 7: 1M Plummer 134.6 / 131.1 / 135.6 ms,
//     200k 21.8 / 22.0 / 23.4, but about one wave, 100k, 9.8 / 9.9 / 10.3 and
//     100k uniform cube 4.31 / 4.67 / 4.95: MORE from a few waves on.
//   3-D, unsoftened (the checks cost registers): 3 / 4 / 5 / 6: 250k 32.3 /
//     30.4 / 31.0 / 32.4 ms, 100k cube 5.2 / 5.0 / 4.6 / -.
//   3-D, split: 4 / 5 / 6 / 7: 250k targets of 1M 28.7 / 27.1 / 26.0 / 25.9 ms,
//     2,000 - / - / 0.89 / 0.91; unsoftened 30k cube 1.12 / 1.07 / 1.10 / -.
//   2-D, softened: 6 / 7 / 8 / 9: 1M 19.7 / 19.5 / 19.2 / 20.0 ms, 100k targets
//     of 1M 4.62 / 4.45 / 4.32 / 4.37, 60k split 1.03 / 0.99 / 0.96 / -; 200k
//     (two waves) 5 / 6: 3.31 / 3.45.
//   2-D, unsoftened: 5 / 6 / 7: 300k 5.08 / 5.02 / 4.88 ms, 60k 1.22 / 1.15 / 1.11.
#ifndef BHUT_FAST_BLOCKS
#define BHUT_FAST_BLOCKS 5
#endif
#ifndef BHUT_FAST_BLOCKS_MORE
#define BHUT_FAST_BLOCKS_MORE 6
#endif
#ifndef BHUT_FAST_BLOCKS_2D
#define BHUT_FAST_BLOCKS_2D 8
#endif
#ifndef BHUT_FAST_BLOCKS_2D_CHECK
#define BHUT_FAST_BLOCKS_2D_CHECK 7
#endif
// Split traversals (split_levels): split while fewer warps than this walk
// and their subtrees hold more nodes than that.  Swept on GB300:
//   warps (ms)            none   6144  12288  24576  49152  98304
//   10k self              1.26   0.34   0.33   0.35   0.34   0.33
//   60k self              6.31   5.08   4.74   4.66   4.55   4.48
//   200k self             23.0      -      -      -   23.3   24.5
//   2,000 targets of 1M   28.8   1.56   1.28   1.20   1.16   1.17
//   100k targets of 1M    21.2   21.2   17.2   16.2   14.5   17.2
//   250k targets of 1M    31.0   31.0   30.7   30.6   29.4   30.4
//   1M self                139      -      -      -    139    181
//   nodes                 4 / 8 / 16 / 32: 10k self 0.42 / 0.35 / 0.34 / 0.33,
//                         1,000 self 0.10 / 0.10 / 0.11 / 0.20
// Self targets that fill the GPU once (kWaveWarps: the wave of the 3-D softened
// kernel, which the others take over) are not split: neighbours then share what
// the walk reads, and a split gives it up.  ms, not split / split, softened and
// not, at 98k, 130k and 195k: uniform cube 4.1 / 3.9, 6.0 / 6.4, 8.7 / 10.6 and
// 4.3 / 4.4, 6.5 / 7.2, 9.0 / 12.3; Plummer 9.2 / 7.9, 14.0 / 12.3, 19.6 / 19.5 and
// 9.5 / 8.9, 14.4 / 13.6, 20.1 / 21.5; 2-D Gaussian 1.67 / 1.83, 2.48 / 2.69, 3.20
// / 3.92.  So the line is right for even distributions and in 2-D, and gives 10 to
// 15 % away just beyond it where the targets' work varies.  External targets vary
// more from group to group, and the shorter walks balance.
#ifndef BHUT_SPLIT_WARPS
#define BHUT_SPLIT_WARPS 49152
#endif
// Trees of one or two long leaves have no nodes to split by: their first two
// levels pay while a warp has this many particles (a split shares a leaf's
// blocks).  Self solves of 500 / 1,000 / 4,000 / 12,000 particles in one or two
// leaves 90 / 138 / 426 / 1,171 us unsplit, 55 / 75 / 149 / 628 split, 40 targets
// 157 / 202 / 478 / 1,230 and 127 / 137 / 219 / 426; by 32 to 128 particles the same.
#ifndef BHUT_SPLIT_PARTICLES
#define BHUT_SPLIT_PARTICLES 64
#endif
// Form "exact" (pairs are dearer, the walk matters less): ms for none / 12501 /
// 25000 / 50001 warps, Plummer: 10k self 10.5 / 2.0 / 2.0 / 2.0, 30k 32.4 /
// 14.6 / 13.7 / 13.3, 60k 62.6 / 42.4 / 40.9 / 40.8, 100k 95.7 / 85.3 / 86.5 /
// 82.5, 200k 208 / 218 / 218 / 213, 2,000 targets of 100k 70.1 / 2.9 / 2.8 /
// 2.8, 100k targets of 200k 121 / 115 / 115 / 125.
#ifndef BHUT_SPLIT_WARPS_EXACT
#define BHUT_SPLIT_WARPS_EXACT 25000
#endif
constexpr int64_t kWaveWarps = 152 * kFastWarps * BHUT_FAST_BLOCKS;   // resident warps
#ifndef BHUT_SPLIT_NODES
#define BHUT_SPLIT_NODES 16
#endif
// The first two levels, shared within a block, pay down to a leaf each: self
// solves of 130 / 300 / 500 points 68 / 87 / 104 us unsplit, 55 / 57 / 68
// split; form "exact" 100 / 300 / 500: 152 / 366 / 566 and 70 / 129 / 179.
#ifndef BHUT_SPLIT_NODES_FIRST
#define BHUT_SPLIT_NODES_FIRST 2
#endif
// ---------------------------------------------------------------------------
// frame (normalisation) derived from the tree's bounding box
// ---------------------------------------------------------------------------
FastFrame frame_of_box(const double* box, int dim)
{
    FastFrame f;
    frame_from_box(box, dim, &f);
    frame_unit_mass(box[6], box[15] != 0.0, &f);
    return f;
}

__global__ void k_ff_particles(const double* __restrict__ sx, const double* __restrict__ sy,
                               const double* __restrict__ sz, const double* __restrict__ sm,
                               int64_t n, int dim, bool fine, FastFrame f,
                               float4* __restrict__ ph, float4* __restrict__ pl)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x) {
        float4 h, l;
        split_grid(sx[i], f.c[0], f.s, fine, h.x, l.x);
        split_grid(sy[i], f.c[1], f.s, fine, h.y, l.y);
        if (dim == 3) split_grid(sz[i], f.c[2], f.s, fine, h.z, l.z);
        else h.z = l.z = 0.0f;
        if (f.unit) { h.w = 1.0f; l.w = 0.0f; }   // every mass is m0: exactly 1 in units of m0
        else split_plain(__dmul_rn(sm[i], f.ms), h.w, l.w);
        ph[i] = h;
        pl[i] = l;
    }
}

__global__ void k_ff_nodes(TreeDev t, bool fine, const double* __restrict__ center,
                           const double* __restrict__ quad, FastFrame f,
                           const float4* __restrict__ ph, NodeCopies o)
{
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < t.m;
         k += (int64_t)gridDim.x * blockDim.x)
        put_node(t, k, f, fine, center, quad, ph, o);
}

// Targets: grid split when inside the box (|u| <= 1), plain split otherwise;
// th.w = 1 marks a target outside the box, tl.w = max |u|.
__global__ void k_ff_targets(const double* __restrict__ tx, const double* __restrict__ ty,
                             const double* __restrict__ tz, int64_t nt, int dim, bool fine,
                             FastFrame f, float4* __restrict__ th,
                             float4* __restrict__ tl)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nt;
         i += (int64_t)gridDim.x * blockDim.x) {
        double u[3] = {__dmul_rn(__dsub_rn(tx[i], f.c[0]), f.s),
                       __dmul_rn(__dsub_rn(ty[i], f.c[1]), f.s),
                       dim == 3 ? __dmul_rn(__dsub_rn(tz[i], f.c[2]), f.s) : 0.0};
        double amax = fmax(fabs(u[0]), fmax(fabs(u[1]), fabs(u[2])));
        bool inside = amax <= 1.0;
        float hh[3], ll[3];
        for (int d = 0; d < 3; d++) {
            if (inside) {
                const float2 p = split_grid_fp64(u[d], fine);
                hh[d] = p.x;
                ll[d] = p.y;
            } else {
                split_plain(u[d], hh[d], ll[d]);
            }
        }
        th[i] = make_float4(hh[0], hh[1], hh[2], inside ? 0.0f : 1.0f);
        tl[i] = make_float4(ll[0], ll[1], ll[2], __double2float_ru(amax));
    }
}

// ---------------------------------------------------------------------------
// the traversal
// ---------------------------------------------------------------------------
struct FastArgs {
    const float4* th;        // target hi (w: outside-box flag); NULL: the particles themselves
    const float4* tl;        // target lo (w: max |u|)
    const double* tx;        // target FP64 (fallbacks)
    const double* ty;
    const double* tz;
    const int32_t* self_id;
    const int32_t* out_idx;
    int64_t nt;
    double theta, eps, G;
    float e2h, e2l;          // (eps * s)^2 as float-float
    double* out;
    unsigned* err;
    unsigned long long* stats;
    int mac;                 // 0: reference criterion, 1: offset criterion (fp32 form)
    float theta2, band2;     // theta^2 and the absolute band of the test on squares (form fast)
};

// leaf_block_soft for the checked path (targets inside the box, softening
// too small to bound r^2 + eps^2 from below: near leaves take pair_ff with
// the range test, pairs below kTinyRCheck in FP64 from the FP64 particle
// arrays).  The split is the same; a lane that works for another lane's
// target also takes that target's FP64 pairs (the target's FP64 coordinates
// are read from memory) and the group adds its FP64 partial sums like the
// float-float ones.  `nfb` counts the FP64 pairs a lane evaluated.
template <int DIM, bool UNIT>
__device__ __forceinline__ void leaf_block_check(unsigned mask, int lane, const float* Th,
                                                 const float* Tl, const FastArgs& a, int64_t base,
                                                 const LeafStage& st, int cn, int first,
                                                 const TreeDev& t, const LeafBox& box, double eps2,
                                                 float* ah, float* al, double* a64, unsigned& nfb)
{
    const unsigned FULL = 0xffffffffu;
    if (mask == 0) return;
    const LaneSplit sp(mask, lane);
    const bool mine = (mask >> lane) & 1u;
    float T[3] = {0.f, 0.f, 0.f}, L[3] = {0.f, 0.f, 0.f};
    split_target<DIM>(sp, Th, Tl, T, L);
    float ph[3] = {0.f, 0.f, 0.f}, pl[3] = {0.f, 0.f, 0.f};
    FarLeaf f;
    const bool far = far_setup<DIM>(T, box, (cn + 1) >> 1, a.e2h, a.e2l, kTinyRCheck, f);
    if (__all_sync(FULL, far || !sp.work)) {
        if (sp.work) far_pairs<DIM, UNIT>(T, L, st, sp.sub, sp.f, cn, f, ph, pl);
        split_add<DIM>(sp, mine, ph, pl, ah, al);
        return;
    }
    unsigned long long fb = 0;
    if (sp.work) {
        // (100,000 particles in one leaf, 3-D / 2-D: rows one by one 49.7 / 40.6
        // ms, by two 46.8 / 39.4; 1M Plummer 137.9 and 136.4)
#pragma unroll 2
        for (int p = sp.sub; 2 * p < cn; p += sp.f) {
#pragma unroll
            for (int o = 0; o < 2; o++) {
                const int q = 2 * p + o;
                if (q >= cn) break;
                float4 h, l;
                st.get(p, o, h, l);
                if (!pair_ff<DIM, false, true>(T, L, h, l, a.e2h, a.e2l, ph, pl)) fb |= 1ull << q;
            }
        }
    }
    split_add<DIM>(sp, mine, ph, pl, ah, al);
    if (!__any_sync(FULL, fb != 0)) return;
    double p64[3] = {0.0, 0.0, 0.0};
    if (fb) {
        const int64_t i = base + sp.owner;
        const double X = a.tx[i], Y = a.ty[i], Z = DIM == 3 ? a.tz[i] : 0.0;
        while (fb) {
            const int gi = first + __ffsll((long long)fb) - 1;
            fb &= fb - 1;
            pair_fp64<DIM>(X, Y, Z, t.sx[gi], t.sy[gi], DIM == 3 ? t.sz[gi] : 0.0, t.sm[gi],
                           eps2, p64);
            nfb++;
        }
    }
    for (int o = sp.f >> 1; o >= 1; o >>= 1) {
#pragma unroll
        for (int c = 0; c < DIM; c++)
            p64[c] = __dadd_rn(p64[c], __shfl_down_sync(FULL, p64[c], o));
    }
#pragma unroll
    for (int c = 0; c < DIM; c++) {
        const double g64 = __shfl_sync(FULL, p64[c], sp.leader);
        if (mine) a64[c] = __dadd_rn(a64[c], g64);
    }
}

// SOFT_PATH (= !FAR && !CHECK): every pair is float-float (no FP64
// fallback); UNIT: leaf pairs skip the mass product (unit masses).
// SPLIT: 2^levels warps share the targets; a warp follows the bits of `path`
// (highest first) through the top `levels` levels and walks the subtree it
// reaches.  A node of those levels is worked on (monopoles, counts) by the warp
// whose remaining bits are zero, a leaf's particles by all that reach it.
// A twig (put_node) that some lane opens is worked on like a leaf: its two
// leaves, always visited by the same lanes, cost one visit, one staging and
// one set of bounds instead of two (1M Plummer 142.7 ms without, 137.0 with,
// 2-D 60k in leaves of 16 1.49 and 1.35).  A box of two leaves is distant less
// often: the larger kFarRatio makes up for it.
template <int DIM, bool FAR, bool CHECK, bool UNIT, bool SPLIT>
__device__ __forceinline__ void walk(const TreeDev& t, const FastTree& ft, const FastArgs& a,
                                     int w, int lane, bool valid, int64_t base, int64_t me_sorted,
                                     const float* Th, const float* Tl, float band_abs, float* ah,
                                     float* al, double* a64, int2 (*stack)[kStackDepth],
                                     LeafStage* stage, unsigned* cnt, bool& overflow,
                                     int levels = 0, int path = 0)
{
    const unsigned FULL = 0xffffffffu;
    const float theta_f = (float)a.theta;
    const double eps2 = __dmul_rn(a.eps, a.eps);
    const int64_t me = base + lane;              // the lane's target
    bool own = !SPLIT || path == 0;              // this warp works on the node
    // The right child of an opened node is visited next, straight from
    // registers; only left children go through the stack.  A visit's three
    // loads (a leaf's box lies where an internal node has its centre of mass)
    // are issued together.
    int node = 0, sp = 0;
    unsigned mask = __ballot_sync(FULL, valid);
    while (true) {
        const bool act = (mask >> lane) & 1u;
        cnt[2] += act && own;
        const int4 hd = ft.nhdr[node];   // (first_child, start, count, flag)
        const float4 nh = ft.nh[node], nl = ft.nl[node];
        const int fc = hd.x;
        LeafBox box{nh, nl};
        unsigned lmask = 0;               // lanes that take the particles [s, s + c)
        int s = hd.y, c = 0;
        if (!hd.w) {                      // mass == 0 skip (bh.py:514)
        } else if (fc < 0) {
            lmask = mask;
            c = hd.z;
            if (SPLIT && levels > 0) {    // runs of whole blocks for the warps that reach it
                const int run = (((c - 1) >> levels) / kStage + 1) * kStage;
                const int first = min(c, (path & ((1 << levels) - 1)) * run);
                s += first;
                c = min(run, c - first);
            }
        } else {
            // The hi parts alone decide outside a band of 2^-14 of d^2 plus
            // 2^-28 (the lo parts move d by delta <= 2^-22, and 2 d delta <=
            // 2^-15 d^2 + 2^15 delta^2); inside it the distance with the lo
            // parts, and inside that one's band FP64.
            float h2 = 0.0f;
#pragma unroll
            for (int k = 0; k < DIM; k++) {
                const float d = __fsub_rn(comp(nh, k), Th[k]);
                h2 = fmaf(d, d, h2);
            }
            const float size_f = __int_as_float(hd.y);
            // (an imported tree may hold negative sizes, which open nothing)
            const float s2 = size_f * fabsf(size_f), td2 = a.theta2 * h2;
            bool open = act && s2 >= td2;
            if (act && (FAR || !(fabsf(s2 - td2) > fmaf(0x1p-14f, td2, a.band2)))) {
                float d2 = 0.0f;
#pragma unroll
                for (int k = 0; k < DIM; k++) {
                    // hi and lo differences, rounded once
                    const float d = __fadd_rn(__fsub_rn(comp(nh, k), Th[k]),
                                              __fsub_rn(comp(nl, k), Tl[k]));
                    d2 = fmaf(d, d, d2);
                }
                // (below 2^-50 the absolute part of the band decides)
                const float dist = d2 > 0x1p-100f ? d2 * rsqrt_mufu(d2) : 0.0f;
                const float td = theta_f * dist;
                const float band = theta_f * fmaf(kBandRel, dist, band_abs);
                if (size_f >= td + band) {
                    open = true;
                } else if (size_f < td - band) {
                    open = false;
                } else {
                    open = open_exact64<DIM>(a.tx[me], a.ty[me], DIM == 3 ? a.tz[me] : 0.0,
                                             t.cm[node], t.size[node], a.theta);
                    cnt[3] += own;
                }
            }
            const unsigned omask = __ballot_sync(FULL, act && open);
            if (act && !open && own) {
                if (!FAR && !CHECK && !(hd.w & kNodeOutside)) {
                    pair_ff_soft<DIM, false>(Th, Tl, nh, nl, a.e2h, a.e2l, ah, al);
                } else if (!FAR && !CHECK) {   // (into the sums: the soft path has no a64)
                    const NodeCM cm = t.cm[node];
                    double f[3] = {0.0, 0.0, 0.0};
                    pair_fp64<DIM>(a.tx[me], a.ty[me], DIM == 3 ? a.tz[me] : 0.0, cm.x, cm.y,
                                   cm.z, cm.w, eps2, f);
#pragma unroll
                    for (int k = 0; k < DIM; k++) {
                        float h, l;
                        split_plain(__ddiv_rn(f[k], ft.frame.conv), h, l);
                        ff_add(ah[k], al[k], h, l);
                    }
                    cnt[4]++;
                } else if ((hd.w & kNodeOutside) ||
                           !pair_ff<DIM, FAR, CHECK>(Th, Tl, nh, nl, a.e2h, a.e2l, ah, al)) {
                    const NodeCM cm = t.cm[node];
                    pair_fp64<DIM>(a.tx[me], a.ty[me], DIM == 3 ? a.tz[me] : 0.0, cm.x, cm.y,
                                   cm.z, cm.w, eps2, a64);
                    cnt[4]++;
                }
                cnt[1]++;
            }
            if (SPLIT && omask && levels > 0) {
                levels--;
                node = fc + ((path >> levels) & 1);
                own = (path & ((1 << levels) - 1)) == 0;
                mask = omask;
                continue;
            }
            if (!FAR && omask && (hd.w & kTwig)) {   // both leaves here
                box = ft.twig[node];
                lmask = omask;
                s = __float_as_int(box.h.w);
                c = twig_left(hd.w) + twig_right(hd.w);
                cnt[2] += open ? 2 : 0;
            } else if (omask) {
                if (sp + 2 > kStackDepth) { overflow = true; break; }
                if (lane == 0) stack[w][sp] = make_int2(fc, (int)omask);
                sp++;
                node = fc + 1;
                mask = omask;
                continue;
            }
        }
        if (c) {
            const bool lact = (lmask >> lane) & 1u;
            if (UNIT) box.c.w = 1.0f;
            for (int b = 0; b < c; b += kStage) {
                const int cn = min(kStage, c - b);
                for (int j = lane; j < cn; j += kWarp)
                    stage[w].put(j, ft.ph[s + b + j], ft.pl[s + b + j]);
                __syncwarp();
                if (lact) {
                    // The target itself (self mode: sorted index `me_sorted`)
                    // sits at zero displacement and adds exactly zero, so it
                    // is not skipped; it is only left out of the pair count
                    // (bh.py:254).
                    cnt[0] += cn - (me_sorted >= s + b && me_sorted < s + b + cn);
                }
                if (!FAR && !CHECK) {
                    leaf_block_soft<DIM, UNIT>(lmask, lane, Th, Tl, stage[w], cn, box, a.e2h, a.e2l,
                                               ah, al);
                } else if (!FAR) {
                    leaf_block_check<DIM, UNIT>(lmask, lane, Th, Tl, a, base, stage[w], cn, s + b, t,
                                                box, eps2, ah, al, a64, cnt[4]);
                } else if (lact) {
                    unsigned long long fb = 0;   // pairs left to FP64 (rare), taken after the loop
#pragma unroll 1
                    for (int q = 0; q < cn; q++) {
                        float4 h, l;
                        stage[w].get(q >> 1, q & 1, h, l);
                        fb |= (unsigned long long)!pair_ff<DIM, FAR, CHECK>(Th, Tl, h, l, a.e2h, a.e2l,
                                                                            ah, al) << q;
                    }
                    while (fb) {
                        const int gi = s + b + __ffsll((long long)fb) - 1;
                        fb &= fb - 1;
                        pair_fp64<DIM>(a.tx[me], a.ty[me], DIM == 3 ? a.tz[me] : 0.0, t.sx[gi],
                                       t.sy[gi], DIM == 3 ? t.sz[gi] : 0.0, t.sm[gi], eps2, a64);
                        cnt[4]++;
                    }
                }
                __syncwarp();
            }
            if (FAR && lact) {   // renormalise once per leaf (ff_add did)
#pragma unroll
                for (int k = 0; k < DIM; k++) {
                    float hsum = __fadd_rn(ah[k], al[k]);
                    al[k] = __fsub_rn(al[k], __fsub_rn(hsum, ah[k]));
                    ah[k] = hsum;
                }
            }
        }
        if (sp == 0) break;
        __syncwarp();
        const int2 e = stack[w][--sp];
        __syncwarp();
        node = e.x;
        mask = (unsigned)e.y;
    }
}

// SOFT: (eps s)^2 >= 2 kTinyR, so a warp of targets inside the box needs no
// small-R test (pair_ff's CHECK).
//
// One warp per 32 targets; with SPLIT (few targets) 2^levels warps per 32
// targets, the block's four among them.  A warp's walk is a chain of
// dependent loads and short loops: it takes its time however few warps run,
// so few targets leave the GPU idle for most of a solve.  Splitting the tree
// shortens the chain itself (figures at BHUT_SPLIT_WARPS).  More warps than
// the GPU holds several times over only repeat the top levels and, with the
// group's warps in different blocks, lose the nodes that they share in L1.
// A block adds its four sums in FP64; with more than four warps per group the blocks' sums go to `partial`
// and k_split_sum adds them (fixed order, no atomics).
template <int DIM, bool SOFT, bool SPLIT, int BLOCKS>
__global__ void __launch_bounds__(kFastThreads, BLOCKS)
k_traverse_fast(TreeDev t, FastTree ft, FastArgs a, int levels, double* __restrict__ partial)
{
    __shared__ int2 stack[kFastWarps][kStackDepth];
    __shared__ LeafStage stage[kFastWarps];
    __shared__ double sum[SPLIT ? kFastWarps : 1][SPLIT ? DIM : 1][kWarp];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const unsigned FULL = 0xffffffffu;
    const FastFrame& fr = ft.frame;
    const double conv = __dmul_rn(fr.conv, a.G);
    const int shares = SPLIT ? (1 << levels) / kFastWarps : 1;   // blocks per group
    const int64_t step = SPLIT ? gridDim.x / shares : (int64_t)gridDim.x * kFastWarps;
    const int share = SPLIT ? (int)(blockIdx.x % (unsigned)shares) : 0;

    for (int64_t g = SPLIT ? blockIdx.x / (unsigned)shares
                           : (int64_t)blockIdx.x * kFastWarps + w;
         g * kWarp < a.nt; g += step) {
        const int64_t base = g * kWarp;
        const int64_t i = base + lane;
        const bool valid = i < a.nt;
        float Th[3] = {0.f, 0.f, 0.f}, Tl[3] = {0.f, 0.f, 0.f};
        bool far = false;
        float amax = 0.f;
        if (valid) {
            // self targets are the sorted particles themselves (inside the box)
            const float4 h = a.th ? a.th[i] : ft.ph[i];
            const float4 l = a.th ? a.tl[i] : ft.pl[i];
            Th[0] = h.x; Th[1] = h.y; Th[2] = h.z;
            Tl[0] = l.x; Tl[1] = l.y; Tl[2] = l.z;
            far = a.th ? h.w != 0.0f : false;
            amax = a.th ? l.w : 1.0f;
        }
        const float band_abs = kBandAbs * (1.0f + amax);
        float ah[3] = {0.f, 0.f, 0.f}, al[3] = {0.f, 0.f, 0.f};
        double a64[3] = {0.0, 0.0, 0.0};
        unsigned cnt[5] = {0, 0, 0, 0, 0};
        // self mode: targets are the sorted particles, target i is particle i
        const int64_t me_sorted = (valid && a.th == nullptr) ? i : -1;
        bool overflow = false;
        const int path = SPLIT ? share * kFastWarps + w : 0;
        if (__any_sync(FULL, far))
            walk<DIM, true, true, false, SPLIT>(t, ft, a, w, lane, valid, base, me_sorted, Th, Tl,
                                                band_abs, ah, al, a64, stack, stage, cnt, overflow,
                                                levels, path);
        else if (fr.unit)
            walk<DIM, false, !SOFT, true, SPLIT>(t, ft, a, w, lane, valid, base, me_sorted, Th, Tl,
                                                 band_abs, ah, al, a64, stack, stage, cnt,
                                                 overflow, levels, path);
        else
            walk<DIM, false, !SOFT, false, SPLIT>(t, ft, a, w, lane, valid, base, me_sorted, Th,
                                                  Tl, band_abs, ah, al, a64, stack, stage, cnt,
                                                  overflow, levels, path);
        if (overflow && lane == 0) atomicOr(a.err, kErrStackOverflow);
        // a share of a split may have had nothing to do: then no counts, and
        // zero sums without the scaling in FP64
        const bool busy = !SPLIT || __any_sync(FULL, (cnt[0] | cnt[1] | cnt[2]) != 0);
        if (a.stats && busy) {
#pragma unroll
            for (int k = 0; k < 5; k++) {
                const unsigned long long v = warp_sum(cnt[k]);
                if (lane == 0 && v) atomicAdd(&a.stats[k], v);
            }
        }
#pragma unroll
        for (int k = 0; k < DIM; k++) {
            double v = 0.0;
            if (busy)
                v = __dadd_rn(__dmul_rn(__dadd_rn((double)ah[k], (double)al[k]), conv),
                              __dmul_rn(a64[k], a.G));
            if (SPLIT) sum[SPLIT ? w : 0][SPLIT ? k : 0][lane] = v;
            else if (valid) a.out[(a.out_idx ? a.out_idx[i] : i) * DIM + k] = v;
        }
        if (SPLIT) {
            __syncthreads();
            if (w < DIM && valid) {
                double v = sum[0][SPLIT ? w : 0][lane];
                for (int u = 1; u < kFastWarps; u++)
                    v = __dadd_rn(v, sum[SPLIT ? u : 0][SPLIT ? w : 0][lane]);
                if (shares > 1) partial[((int64_t)share * a.nt + i) * DIM + w] = v;
                else a.out[(a.out_idx ? a.out_idx[i] : i) * DIM + w] = v;
            }
            __syncthreads();
        }
    }
}

// kSumRows threads per output, each with every kSumRows-th share: one thread
// for all of 256 shares took 32 us for 2,000 targets.  PAIRS (form exact): each
// with a run of shares, added in pairs as the tree's levels are.
constexpr int kSumRows = 8;
template <bool PAIRS>
__global__ void __launch_bounds__(kWarp * kSumRows)
k_split_sum(const double* __restrict__ partial, int64_t nt, int dim, int shares,
            const int32_t* __restrict__ out_idx, double* __restrict__ out)
{
    __shared__ double part[kSumRows][kWarp];
    for (int64_t base = blockIdx.x * (int64_t)kWarp; base < nt * dim;
         base += (int64_t)gridDim.x * kWarp) {
        const int64_t j = base + threadIdx.x;
        double v = 0.0;
        if (PAIRS && j < nt * dim) {
            const int run = max(shares / kSumRows, 1), y0 = threadIdx.y * run;
            double wait[kTopLevels];   // sums of whole runs of 2^k shares
            for (int y = 0; y0 < shares && y < run; y++) {
                v = partial[(int64_t)(y0 + y) * nt * dim + j];
                int k = 0;
                for (; (y >> k) & 1; k++) v = __dadd_rn(wait[k], v);
                wait[k] = v;
            }
        } else if (j < nt * dim) {
#pragma unroll 8
            for (int y = threadIdx.y; y < shares; y += kSumRows)
                v = __dadd_rn(v, partial[(int64_t)y * nt * dim + j]);
        }
        part[threadIdx.y][threadIdx.x] = v;
        __syncthreads();
        if (threadIdx.y == 0 && j < nt * dim) {
            if (PAIRS) {
                double p[kSumRows];
                for (int y = 0; y < kSumRows; y++) p[y] = part[y][threadIdx.x];
#pragma unroll
                for (int o = 1; o < kSumRows; o *= 2)
#pragma unroll
                    for (int y = 0; y < kSumRows; y += 2 * o) p[y] = __dadd_rn(p[y], p[y + o]);
                v = p[0];
            } else {
                for (int y = 1; y < min(kSumRows, shares); y++)
                    v = __dadd_rn(v, part[y][threadIdx.x]);
            }
            const int64_t i = j / dim;
            out[(out_idx ? out_idx[i] : i) * dim + j % dim] = v;
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// form "fp32": the precision form.  Pair terms, monopoles and the opening
// test in FP32 on hi + lo displacements (each difference exact, rounded
// once); per-target sums Kahan-compensated: every monopole, and every leaf
// block of at most 32 pair terms (summed in FP32 first), is one Kahan step.
// Walk and rows are in fast.cuh (walk_f32, rows_f32), with the figures.  2M
// galaxy, theta 0.7, leaf 16: 119 -> 101 ms with two sources to a row, the
// opening test on squares, leaf pairs in one visit and children tested
// together.  Prefetching the next nodes' headers: 122 to 126 ms, not kept.
// FP64 stays in the tree build (bounding box, Morton keys, masses and
// centres of mass, quadrupoles) and in the final scaling.
// ---------------------------------------------------------------------------
// Resident blocks per SM: 8 / 9 / 10 / 11 at 2M galaxy, theta 0.7, leaf 16:
// 103.6 / 101.2 / 104.5 / 125 ms (more blocks leave fewer registers, and less
// L1 beside the stages and stacks).
#ifndef BHUT_F32_BLOCKS
#define BHUT_F32_BLOCKS 9
#endif
template <int DIM>
__global__ void __launch_bounds__(kFastThreads, BHUT_F32_BLOCKS)
k_traverse_fp32(TreeDev t, FastTree ft, FastArgs a)
{
    __shared__ StackEntry stack[kFastWarps][kStackDepth];
    __shared__ LeafStage stage[kFastWarps];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const unsigned FULL = 0xffffffffu;
    const double conv = __dmul_rn(ft.frame.conv, a.G);
    const OpenF32 opener(a.theta, a.mac);
    for (int64_t base = ((int64_t)blockIdx.x * kFastWarps + w) * kWarp; base < a.nt;
         base += (int64_t)gridDim.x * kFastWarps * kWarp) {
        const int64_t i = base + lane;
        const bool valid = i < a.nt;
        float T[3] = {0.f, 0.f, 0.f}, Tl[3] = {0.f, 0.f, 0.f};
        bool outside = false;
        if (valid) {
            const float4 h = a.th ? a.th[i] : ft.ph[i];
            const float4 l = a.th ? a.tl[i] : ft.pl[i];
            T[0] = h.x; T[1] = h.y; T[2] = h.z;
            Tl[0] = l.x; Tl[1] = l.y; Tl[2] = l.z;
            outside = a.th && h.w != 0.0f;
        }
        outside = __any_sync(FULL, outside);
        float acc[3] = {0.f, 0.f, 0.f}, cmp[3] = {0.f, 0.f, 0.f};
        unsigned cnt[5] = {0, 0, 0, 0, 0};
        const int me = valid && a.th == nullptr ? (int)i : -1;
        bool overflow = false;
        WarpStack<0> st(stack[w], lane);
        walk_f32<DIM>(ft, 0, lane, valid, me, outside, ft.frame.unit != 0 && !outside, opener,
                      a.e2h, T, Tl, acc, cmp, st, stage[w], cnt, overflow);
        if (overflow && lane == 0) atomicOr(a.err, kErrStackOverflow);
        if (a.stats) {
#pragma unroll
            for (int k = 0; k < 3; k++) {
                const unsigned long long v = warp_sum(cnt[k]);
                if (lane == 0 && v) atomicAdd(&a.stats[k], v);
            }
        }
        if (valid) {
            const int64_t o = a.out_idx ? a.out_idx[i] : i;
#pragma unroll
            for (int k = 0; k < DIM; k++)   // Kahan sum: value = sum - compensation
                a.out[o * DIM + k] = __dmul_rn(__dsub_rn((double)acc[k], (double)cmp[k]), conv);
        }
    }
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
int launch_fast_prepare(const FastFrame& frame, bool fine, const TreeDev& t, const double* center,
                        const double* quad, float4* ph, float4* pl, const NodeCopies& o,
                        cudaStream_t s)
{
    k_ff_particles<<<grid_for(t.n, 256), 256, 0, s>>>(t.sx, t.sy, t.sz, t.sm, t.n, t.dim, fine,
                                                      frame, ph, pl);
    k_ff_nodes<<<grid_for(t.m, 256), 256, 0, s>>>(t, fine, center, quad, frame, ph, o);
    BHUT_CUDA(cudaGetLastError());
    note_launches(2);
    return kOk;
}

int launch_fast_targets(const double* tx, const double* ty, const double* tz, int64_t nt, int dim,
                        bool fine, const FastFrame& frame, float4* th, float4* tl, cudaStream_t s)
{
    k_ff_targets<<<grid_for(nt, 256), 256, 0, s>>>(tx, ty, tz, nt, dim, fine, frame, th, tl);
    BHUT_CUDA(cudaGetLastError());
    note_launches(1);
    return kOk;
}

int launch_split_sum(const double* partial, int64_t nt, int dim, int shares, bool pairs,
                     const int32_t* out_idx, double* out, cudaStream_t s)
{
    const auto kernel = pairs ? k_split_sum<true> : k_split_sum<false>;
    kernel<<<grid_for(nt * dim, kWarp), dim3(kWarp, kSumRows), 0, s>>>(partial, nt, dim, shares,
                                                                      out_idx, out);
    BHUT_CUDA(cudaGetLastError());
    note_launches(1);
    return kOk;
}

// Whether a tree of so many nodes has work for another level of a split.
static bool splits_further(int64_t nodes, int levels)
{
    return levels < kTopLevels &&
           (nodes >> levels) > (levels < 2 ? BHUT_SPLIT_NODES_FIRST : BHUT_SPLIT_NODES);
}

int top_levels(int64_t nodes)
{
    int levels = 0;
    while (splits_further(nodes, levels)) levels++;
    return levels;
}

// Levels of the tree to split a traversal of nt targets by (0: none, else
// 2 to kTopLevels), and the doubles of `partial` it needs.
int split_levels(int64_t nt, int64_t nodes, int64_t particles, bool self, bool exact)
{
    const int64_t groups = (nt + kWarp - 1) / kWarp;
    if (self && groups >= (exact ? 2 : 1) * kWaveWarps) return 0;
    const int64_t warps = exact ? BHUT_SPLIT_WARPS_EXACT : BHUT_SPLIT_WARPS;
    int levels = 0;
    while ((groups << levels) < warps &&
           (splits_further(nodes, levels) ||
            (!exact && levels < 2 && (particles >> levels) > 2 * BHUT_SPLIT_PARTICLES)))
        levels++;
    return levels < 2 ? 0 : levels;
}

int64_t split_partial_doubles(int64_t nt, int dim, int levels)
{
    const int64_t shares = (1 << levels) / kFastWarps;
    return levels > 0 && shares > 1 ? shares * nt * dim : 0;
}

int launch_traverse_fast(const TreeDev& t, const FastTree& ft, const float4* th, const float4* tl,
                         const double* tx, const double* ty, const double* tz,
                         const int32_t* self_id, const int32_t* out_idx, int64_t nt, double theta,
                         double eps, double G, double eps_scaled_sq, double* out, unsigned* err,
                         unsigned long long* stats, cudaStream_t s, bool fp32, int mac,
                         int levels, double* partial)
{
    if (nt <= 0) return kOk;
    FastArgs a;
    a.th = th; a.tl = tl; a.tx = tx; a.ty = ty; a.tz = tz;
    a.self_id = self_id; a.out_idx = out_idx; a.nt = nt;
    a.theta = theta; a.eps = eps; a.G = G;
    a.e2h = (float)eps_scaled_sq;
    a.e2l = (float)(eps_scaled_sq - (double)a.e2h);
    a.out = out; a.err = err; a.stats = stats; a.mac = mac;
    // A theta whose products would leave the range in which they keep 2^-14 gets an
    // infinite band: the squares then decide nothing.  (Kernel arguments: chosen
    // in the walk, the band cost a register and 0.5 to 1 % of the time.)
    const float tf = (float)theta;
    a.theta2 = tf * tf;
    a.band2 = tf == 0.0f || (tf >= 0x1p-30f && tf <= 0x1p+30f) ? 0x1p-28f * a.theta2 : INFINITY;
    int64_t warps = (nt + kWarp - 1) / kWarp;
    unsigned grid = grid_for(warps, kFastWarps, 152u * 64u);
    if (fp32) {
        if (t.dim == 3) k_traverse_fp32<3><<<grid, kFastThreads, 0, s>>>(t, ft, a);
        else k_traverse_fp32<2><<<grid, kFastThreads, 0, s>>>(t, ft, a);
    } else {
        const bool soft = a.e2h >= 2.0f * kTinyR;
        constexpr int B = BHUT_FAST_BLOCKS, MORE = BHUT_FAST_BLOCKS_MORE;
        constexpr int B2 = BHUT_FAST_BLOCKS_2D, C2 = BHUT_FAST_BLOCKS_2D_CHECK;
        const bool d3 = t.dim == 3;
        const int shares = levels > 0 ? (1 << levels) / kFastWarps : 0;
        const unsigned g = shares ? (unsigned)warps * (unsigned)shares : grid;
        const auto kernel =
            shares                    ? (soft ? (d3 ? k_traverse_fast<3, true, true, MORE>
                                                    : k_traverse_fast<2, true, true, B2>)
                                              : (d3 ? k_traverse_fast<3, false, true, B>
                                                    : k_traverse_fast<2, false, true, C2>))
            : !soft                   ? (d3 ? k_traverse_fast<3, false, false, B>
                                            : k_traverse_fast<2, false, false, C2>)
            : warps >= 3 * kWaveWarps ? (d3 ? k_traverse_fast<3, true, false, MORE>
                                            : k_traverse_fast<2, true, false, B2>)
                                      : (d3 ? k_traverse_fast<3, true, false, B>
                                            : k_traverse_fast<2, true, false, B>);
        kernel<<<g, kFastThreads, 0, s>>>(t, ft, a, levels, partial);
        if (shares > 1) BHUT_TRY(launch_split_sum(partial, nt, t.dim, shares, false, out_idx, out, s));
    }
    BHUT_CUDA(cudaGetLastError());
    note_launches(1);
    return kOk;
}

}  // namespace bhut
