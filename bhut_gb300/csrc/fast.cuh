// Device arithmetic shared by the single-tree and batched traversals:
// normalisation frames, the grid-aligned hi/lo split of coordinates, the
// float-float pair term (form "fast"), the FP32 pair term (form "fp32"),
// the FP64 pair term and the exact FP64 opening test used as fallbacks.
#pragma once
#include "tree.cuh"

// Accumulation two-sum of pair_ff_soft: 0 = FastTwoSum on the operands
// ordered by magnitude (ALU compare and selects), 1 = Knuth's TwoSum (six
// FP32 operations).  Both are exact; build-time switch for measurements.
#ifndef BHUT_FF_KNUTH_ACC
#define BHUT_FF_KNUTH_ACC 0
#endif

namespace bhut {

// leaf_block_soft: leaf visits with at most kSplitMaxK active lanes are split
// across the idle lanes.  (The FP32 form's pair term is too cheap for the
// split to pay, 63.9-64.1 ms against 62.7 ms unsplit at 1M Plummer, so it
// keeps one lane per target.)
constexpr int kSplitMaxK = 16;
static_assert(kSplitMaxK <= 16, "a split gives every active target at least two lanes");

// A displacement is known to about 2^-48 (normalised units), so a pair's
// relative error is about 2^-48 / sqrt(R), R = r^2 + eps^2.
// Softened path: every R is at least eps^2, and the range test is compiled
// out when (eps s)^2 >= 2 kTinyR.
constexpr float kTinyR = 0x1p-34f;
// Checked path (small or no softening): R below this -> FP64 pair, so a
// float-float pair's relative error stays below 2^-35.
constexpr float kTinyRCheck = 0x1p-26f;
constexpr float kHugeR = 0x1p+100f;    // r^2 above this -> FP64 pair
constexpr float kBandRel = 0x1p-18f;   // opening-test error band, relative part
constexpr float kBandAbs = 0x1p-40f;   // ... absolute part per unit of (1 + |target|)

// (Only single roundings and powers of two: host and device agree bit for bit.)
static __host__ __device__ inline void frame_from_box(const double* box, int dim, FastFrame* f)
{
    double h = 0.0;
    for (int d = 0; d < 3; d++) f->c[d] = 0.0;
    for (int d = 0; d < dim; d++) {
        f->c[d] = (box[d] + box[3 + d]) * 0.5;
        double e = (box[3 + d] - box[d]) * 0.5;
        h = e > h ? e : h;
    }
    if (!(h > 0.0)) h = 1.0;
    // Map the box into [-1/2, 1/2]: a refit may move particles to 1.1x the
    // root box (bhut/tree/refit.py:236-249) and targets inside [-1, 1] are
    // still on the grid; every hi difference then stays below 2 and is exact.
    int ex;
    frexp(h, &ex);                      // h <= 2^ex
    f->s = ldexp(1.0, -ex - 1);
    double mm = box[6];
    int em = 0;
    if (mm > 0.0) frexp(mm, &em);       // |m| <= 2^em
    f->ms = ldexp(1.0, -em);
    f->conv = ldexp(1.0, em - 2 * ex - 2);  // normalised -> physical acceleration (s^2 / ms)
    f->unit = 0;
}

// Every particle has the same positive mass m0 (flag set by the
// bounding-box kernel): masses are measured in units of m0, so a particle's
// normalised mass is exactly 1 and a node's is M / m0 (FP64, then split hi +
// lo).
static __host__ __device__ inline void frame_unit_mass(double m0, bool uniform, FastFrame* f)
{
    if (!uniform || !(m0 > 0x1p-1000 && m0 < 0x1p+1000)) return;
    f->ms = 1.0 / m0;
    f->conv = m0 * f->s * f->s;   // s a power of two: exact
    f->unit = 1;
}


// hi on the 2^-23 grid (differences of hi parts are exact in FP32 for |u| <=
// 1) and lo the rest, |lo| <= 2^-24:
//  * rounded to FP32 (`fine`, form "fast"): u is represented to within 2^-49,
//    differences of lo parts are rounded to within 2^-48;
//  * on the 2^-47 grid (form "fp32"): u to within 2^-48, differences exact.
// The grid's own error was the largest of a float-float solve (200k Plummer,
// softening 0.01: 9.6e-13 relative L2 against IEEE FP64, rounded lo parts
// 5.5e-13); the FP32 form, at 3e-8, keeps the grid and its results.
static __device__ __noinline__ float2 split_grid_fp64(double u, bool fine)
{
    double H = rint(__dmul_rn(u, 8388608.0));
    double hd = __dmul_rn(H, 1.0 / 8388608.0);
    double r = __dsub_rn(u, hd);
    if (!fine)
        r = __dmul_rn(rint(__dmul_rn(r, 140737488355328.0)), 1.0 / 140737488355328.0);   // 2^47
    return make_float2(__double2float_rn(hd), __double2float_rn(r));
}

// The same for u = v s, s a power of two, in integers: |u| < 2 as a fixed-point
// number F with 62 fraction bits (bits below them kept as a sticky last bit),
// rounded to 23 of them for hi, the rest converted or rounded for lo.  False:
// u is not such a number, or so small a rest that the dropped bits count.
// The copies of 1M particles took 63 us with the eight FP64 instructions of the
// general form per coordinate, all of it on the FP64 pipe; a rebuild of 1M with
// 2,000 targets went from 1.39 to 1.30 ms.
static __host__ __device__ __forceinline__ bool split_grid_int(uint64_t v, uint64_t s, bool fine,
                                                               float& h, float& l)
{
    const int ev = (int)(v >> 52) & 0x7ff, es = (int)(s >> 52) & 0x7ff;
    const int k = ev + es - 2 * 1023 + 10;   // |u| = m 2^(k - 62)
    if (ev == 0 || es == 0 || k > 10 || k < -40) return false;
    const uint64_t m = (v & 0xfffffffffffffull) | 0x10000000000000ull;
    uint64_t F = m << (k > 0 ? k : 0);
    if (k < 0) F = (m >> -k) | (uint64_t)((m & ((1ull << -k) - 1)) != 0);
    const uint64_t H = (F + ((1ull << 38) - 1) + ((F >> 39) & 1)) >> 39;
    int64_t r = (int64_t)(F - (H << 39));
    if (k < 0 && r > -(1 << 25) && r < (1 << 25)) return false;
    const float sign = v >> 63 ? -1.0f : 1.0f;
    h = sign * ((float)(int)H * 0x1p-23f);
    if (fine) {
        l = sign * ((float)r * 0x1p-62f);
    } else {
        r = (r + ((1 << 14) - 1) + ((r >> 15) & 1)) >> 15;   // to 2^-47, ties to even
        l = sign * ((float)(int)r * 0x1p-47f);
    }
    return true;
}

// hi and lo of (x - c) s in a frame.
static __device__ __forceinline__ void split_grid(double x, double c, double s, bool fine, float& h,
                                                  float& l)
{
    const double v = __dsub_rn(x, c);
    if (!split_grid_int((uint64_t)__double_as_longlong(v), (uint64_t)__double_as_longlong(s), fine, h,
                        l)) {
        const float2 p = split_grid_fp64(__dmul_rn(v, s), fine);
        h = p.x;
        l = p.y;
    }
}

// Sum of a 32-bit count over the warp (two reductions, so that it cannot wrap).
static __device__ __forceinline__ unsigned long long warp_sum(unsigned v)
{
    const unsigned lo = __reduce_add_sync(0xffffffffu, v & 0xffffu);
    const unsigned hi = __reduce_add_sync(0xffffffffu, v >> 16);
    return lo + ((unsigned long long)hi << 16);
}

// A node's header flag: 0 without mass (skipped), 1, or 3 when its centre of
// mass lies outside the box (masses of both signs): its coordinates are not
// on the grid and its monopole is taken in FP64.
static __device__ __forceinline__ int node_flag(const NodeCM& c, const float4& h)
{
    const bool out = !(fabsf(h.x) <= 1.0f && fabsf(h.y) <= 1.0f && fabsf(h.z) <= 1.0f);
    return c.w == 0.0 ? 0 : (out ? 3 : 1);
}

static __device__ __forceinline__ void split_plain(double u, float& h, float& l)
{
    h = __double2float_rn(u);
    l = __double2float_rn(__dsub_rn(u, (double)h));
}


// ---------------------------------------------------------------------------
// float-float pair term
// ---------------------------------------------------------------------------
// Error of s = fl(a + b) (Knuth's TwoSum).
static __device__ __forceinline__ float two_sum_err(float a, float b, float s)
{
    float bb = __fsub_rn(s, a);
    return __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
}

// MUFU reciprocal square root, flush-to-zero (one instruction; callers pass
// normal, positive arguments only).
static __device__ __forceinline__ float rsqrt_mufu(float x)
{
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

static __device__ __forceinline__ float comp(const float4& v, int k)
{
    return k == 0 ? v.x : (k == 1 ? v.y : v.z);
}

// Adds G-less m * (x_src - x_tgt) / (|dx|^2 + eps^2)^(3/2), normalised
// units, to (ah, al).  Returns false when the pair must go to FP64; it then
// adds exactly zero (the term is computed on a stand-in R and discarded with
// selects, so the pair loop has no branch).
//
// d = hi_src - hi_tgt is exact on the grid and l = lo_src - lo_tgt is small
// (|l| <= 2^-23, rounded to 2^-48), so (d, l) is renormalised with FastTwoSum into (gh, gl),
// |gl| <= ulp(gh) / 2; every later product of a float-float with g then
// keeps ~2^-47 relative accuracy.  A pair at zero displacement (the target
// itself, or a duplicate) contributes exactly zero, as in the reference.
//
// CHECK = false: the caller guarantees R >= kTinyR for every pair (a target
// inside the box and a softening with (eps s)^2 >= 2 kTinyR: R >= eps^2 up to
// the 2^-20 relative error of the error terms), so the test and its selects
// are compiled out and the result is the same bit for bit.
template <int DIM, bool FAR, bool CHECK = true>
__device__ __forceinline__ bool pair_ff(const float* Th, const float* Tl, float4 sh, float4 sl,
                                        float e2h, float e2l, float* ah, float* al)
{
    float gh[3], gl[3];
#pragma unroll
    for (int k = 0; k < DIM; k++) {
        const float xh = comp(sh, k);
        const float d = __fsub_rn(xh, Th[k]);        // exact on the grid
        float l = __fsub_rn(comp(sl, k), Tl[k]);
        if (FAR) l = __fadd_rn(l, two_sum_err(xh, -Th[k], d));
        const float h = __fadd_rn(d, l);             // FastTwoSum(d, l), |l| <= |d| or d == 0
        gl[k] = __fsub_rn(l, __fsub_rn(h, d));
        gh[k] = h;
    }
    // R = |g|^2 + eps^2: squares error-free, cross terms 2 gh gl in FP32
    float s = __fmul_rn(gh[0], gh[0]);
    float lo = __fmaf_rn(gh[0], gh[0], -s);
    float c = __fmul_rn(gh[0], gl[0]);
#pragma unroll
    for (int k = 1; k < DIM; k++) {
        const float p = __fmul_rn(gh[k], gh[k]);
        const float q = __fmaf_rn(gh[k], gh[k], -p);
        const float t = __fadd_rn(s, p);
        lo = __fadd_rn(lo, __fadd_rn(two_sum_err(s, p, t), q));
        s = t;
        c = __fmaf_rn(gh[k], gl[k], c);
    }
    {
        const float t = __fadd_rn(s, e2h);
        lo = __fadd_rn(lo, __fadd_rn(two_sum_err(s, e2h, t), __fmaf_rn(2.0f, c, e2l)));
        s = t;
    }
    const float Rs = __fadd_rn(s, lo);
    // |dx| <= 2 inside the box: only FAR targets can exceed kHugeR
    const bool ok = FAR ? (Rs >= kTinyRCheck && Rs <= kHugeR) : (!CHECK || Rs >= kTinyRCheck);
    const float Rh = ok ? Rs : 1.0f;
    const float Rl = ok ? __fsub_rn(lo, __fsub_rn(Rs, s)) : 0.0f;
    // w = R^(-3/2): y ~ R^(-1/2); e = 1 - R y^2 exactly enough;
    // w = y^3 (1 - e)^(-3/2) = y^3 (1 + 3e/2 + 15e^2/8 + O(e^3))
    const float y = rsqrt_mufu(Rh);                  // Rh >= kTinyRCheck: normal
    const float Y = __fmul_rn(y, y);
    const float Ye = __fmaf_rn(y, y, -Y);
    const float e = -__fmaf_rn(Rh, Ye, __fmaf_rn(Rl, Y, __fmaf_rn(Rh, Y, -1.0f)));
    const float W = __fmul_rn(Y, y);
    const float We = __fmaf_rn(Ye, y, __fmaf_rn(Y, y, -W));
    const float corr = __fmul_rn(e, __fmaf_rn(1.875f, e, 1.5f));
    const float wh = W;
    const float wl = __fmaf_rn(W, corr, We);
    // f = m w (zero for a pair left to FP64)
    const float mh = ok ? sh.w : 0.0f, ml = ok ? sl.w : 0.0f;
    const float fh = __fmul_rn(mh, wh);
    const float fl = __fmaf_rn(mh, wl, __fmaf_rn(ml, wh, __fmaf_rn(mh, wh, -fh)));
#pragma unroll
    for (int k = 0; k < DIM; k++) {
        const float Fh = __fmul_rn(fh, gh[k]);
        const float Fl = __fmaf_rn(fh, gl[k], __fmaf_rn(fl, gh[k], __fmaf_rn(fh, gh[k], -Fh)));
        const float t = __fadd_rn(ah[k], Fh);
        const float err = two_sum_err(ah[k], Fh, t);
        ah[k] = t;
        al[k] = __fadd_rn(al[k], __fadd_rn(err, Fl));
    }
    return ok;
}

// The float-float pair term for a target inside the box when the softening
// bounds R = |g|^2 + eps^2 from below ((eps s)^2 >= 2 kTinyR: no pair can go
// to FP64).  Same inputs and result as pair_ff<DIM, false, false> up to the
// last bits, with fewer operations:
//  * the squares and eps^2 are non-negative, so each of the three additions
//    of R's high part is Dekker's FastTwoSum on (max, min) (two min/max on
//    the ALU pipe and three FP32 operations instead of Knuth's six);
//  * R stays unnormalised as s + lo (|lo| <= 2^-22 s): the rsqrt is taken of
//    s and the correction term e = 1 - (s + lo) y^2 absorbs lo;
//  * w = y^3 (1 + 3e/2): |e| <= 2^-20.4 (MUFU error plus |lo| / s), so the
//    dropped 15e^2/8 term is below 2^-39.9 of the pair, and in practice far
//    below the 2^-48 representation of the coordinates (|g| is near-pair
//    sized: ~2^-36 relative for a leaf pair);
//  * the accumulation stays an exact two-sum, written as FastTwoSum on the
//    operands ordered by magnitude (one compare and two selects on the ALU
//    pipe, three FP32 operations);
//  * UNIT: masses are in units of the common particle mass (every particle
//    has mass exactly 1), so f = w and the mass product is skipped.
template <int DIM, bool UNIT>
__device__ __forceinline__ void pair_ff_soft(const float* Th, const float* Tl, float4 sh,
                                             float4 sl, float e2h, float e2l, float* ah, float* al)
{
    float gh[3], gl[3], p[3], q[3];
#pragma unroll
    for (int k = 0; k < DIM; k++) {
        const float d = __fsub_rn(comp(sh, k), Th[k]);   // exact on the grid
        const float l = __fsub_rn(comp(sl, k), Tl[k]);
        const float h = __fadd_rn(d, l);                  // FastTwoSum(d, l)
        gl[k] = __fsub_rn(l, __fsub_rn(h, d));
        gh[k] = h;
        p[k] = __fmul_rn(h, h);
        q[k] = __fmaf_rn(h, h, -p[k]);                   // exact square error
    }
    float c = __fmul_rn(gh[0], gl[0]);
#pragma unroll
    for (int k = 1; k < DIM; k++) c = __fmaf_rn(gh[k], gl[k], c);
    // s = ((eps^2 + p0) + p1) + p2, each error exact
    float s = e2h, lo = __fmaf_rn(2.0f, c, e2l);
#pragma unroll
    for (int k = 0; k < DIM; k++) {
        const float a = fmaxf(s, p[k]), b = fminf(s, p[k]);
        const float t = __fadd_rn(a, b);
        lo = __fadd_rn(lo, __fadd_rn(__fsub_rn(b, __fsub_rn(t, a)), q[k]));
        s = t;
    }
    // y ~ s^(-1/2); A = (s + lo) y^2 - 1 = -e to ~2^-46
    const float y = rsqrt_mufu(s);                    // s >= eps^2 > 0: normal
    const float Y = __fmul_rn(y, y);
    const float Ye = __fmaf_rn(y, y, -Y);
    const float A = __fmaf_rn(s, Ye, __fmaf_rn(lo, Y, __fmaf_rn(s, Y, -1.0f)));
    const float W = __fmul_rn(Y, y);
    const float We = __fmaf_rn(Ye, y, __fmaf_rn(Y, y, -W));
    const float wl = __fmaf_rn(__fmul_rn(W, -1.5f), A, We);   // y^3 (1 + 1.5 e) - W
    float fh = W, fl = wl;
    if (!UNIT) {
        const float mh = sh.w, ml = sl.w;
        fh = __fmul_rn(mh, W);
        fl = __fmaf_rn(mh, wl, __fmaf_rn(ml, W, __fmaf_rn(mh, W, -fh)));
    }
#pragma unroll
    for (int k = 0; k < DIM; k++) {
        const float Fh = __fmul_rn(fh, gh[k]);
        const float Fl = __fmaf_rn(fh, gl[k], __fmaf_rn(fl, gh[k], __fmaf_rn(fh, gh[k], -Fh)));
        const float t = __fadd_rn(ah[k], Fh);
#if BHUT_FF_KNUTH_ACC
        const float err = two_sum_err(ah[k], Fh, t);
#else
        const bool sw = fabsf(Fh) > fabsf(ah[k]);
        const float big = sw ? Fh : ah[k], small = sw ? ah[k] : Fh;
        const float err = __fsub_rn(small, __fsub_rn(t, big));
#endif
        ah[k] = t;
        al[k] = __fadd_rn(al[k], __fadd_rn(err, Fl));
    }
}

// Float-float (ah, al) += (bh, bl): TwoSum of the high parts, the low parts
// added to its error, renormalised by FastTwoSum.
static __device__ __forceinline__ void ff_add(float& ah, float& al, float bh, float bl)
{
    const float s = __fadd_rn(ah, bh);
    const float e = __fadd_rn(two_sum_err(ah, bh, s), __fadd_rn(al, bl));
    const float h = __fadd_rn(s, e);
    al = __fsub_rn(e, __fsub_rn(h, s));
    ah = h;
}

// Position of the set bit of rank r (0-based, from the least significant
// bit) of m; m must have more than r bits set.
static __device__ __forceinline__ int nth_set_bit(unsigned m, int r)
{
    int pos = 0;
#pragma unroll
    for (int w = 16; w >= 1; w >>= 1) {
        const int c = __popc(m & ((1u << w) - 1u));
        if (r >= c) {
            r -= c;
            m >>= w;
            pos += w;
        }
    }
    return pos;
}

// ---------------------------------------------------------------------------
// float-float pair term of a distant leaf
// ---------------------------------------------------------------------------
// The bounding box of a leaf gives a target bounds on everything the pair
// term adds up, and a bound makes a compensated sum cheap: with an
// accumulator s known to be at least as large as the term, t = fma(a, b, s)
// has t - s exact (Sterbenz) and fma(a, b, -(t - s)) is the exact rounding
// error -- three FP32 operations to add a PRODUCT without error, no ordering
// of the operands and no separate two-product.  The biases cost bits where
// the bounds are loose, so the term serves leaves whose max R is at most
// kFarRatio times their min R.
//   * r^2 starts at s0 >= max R (subtracted again exactly: R <= s0), so its
//     three squares cost 5 operations each (with the cross term of the lo
//     parts) instead of 9 and two min/max;
//   * the leaf's force sums start at +-B, B a power of two above twice any
//     term plus what the terms can take off it, on the side of the box
//     (terms of the other sign come from |d_k| <= h_k - |g_k| only); B comes
//     off exactly after the leaf.  6 operations per component instead of 9 and
//     three of the ALU pipe;
//   * the displacement stays (d, l) without renormalisation: |l| <= 2^-23,
//     and the products with l are rounded once at 2^-24 of themselves, i.e.
//     2^-47 / D of the pair -- the error that the coordinates have anyway;
//   * neither r^2 = (R0, lo) nor y is renormalised: y is the rsqrt of 2 r^2 / 3,
//     Y the rounded y^2 and taken as it is.  A = r^2 Y - 3/2 and b = y^2 - Y
//     are small, and the cube of the root is Y y (1 - A) - b y / 2 with no
//     constant left (A^2 terms below 2^-42); -y / 2 costs an ALU addition.
//     The leaf's sums carry the factor (3/2)^(3/2), taken off at its end.
// 53 FP32 operations and one MUFU per pair with unit masses, against 77, 15
// on the ALU pipe and one MUFU of pair_ff_soft.  (56, with r^2 renormalised
// and b in A: 1M Plummer 134.1 ms, 250k targets 25.8, 100k cube without
// softening 5.07; 53: 133.1, 24.9, 4.86; errors against FP64 the same.)
constexpr float kFarScale = 0.54433105395181735517;   // (2/3)^(3/2), float-float
constexpr float kFarScaleLo = 0.54433105395181735517 - (double)kFarScale;

// Two sources go through each operation together (f32x2: FADD2 / FFMA2, the
// same IEEE operations; a difference is an FFMA2 by -1): half the issue slots
// and two independent chains per lane.
// kFarRatio 16 / 32 / 64 / 256: 1M Plummer 137.0 / 134.8 / 133.6 / 132.4 ms;
// error against FP64 sums in 2-D, 60k, 1.3e-12 / 1.3e-12 / 2.2e-12 / 6.9e-12
// (2.2e-12 with pair_ff_soft for every leaf).
constexpr float kFarRatio = 32.0f;
struct FarLeaf {
    float s0;      // bias of r^2, at least max R
    float si, li;  // s0 + eps^2 as si + li
    float b[3];    // bias of the force sums
};

// Up to kStage sources staged for a warp, two to a row: source 2p in the even
// and 2p + 1 in the odd components.
constexpr int kStage = 2 * kWarp;
struct LeafStage {
    float4 a[kStage / 2];   // (x hi, x hi', y hi, y hi')
    float4 b[kStage / 2];   // (x lo, x lo', y lo, y lo')
    float4 c[kStage / 2];   // (z hi, z hi', z lo, z lo')
    float4 d[kStage / 2];   // (m hi, m hi', m lo, m lo')
    __device__ __forceinline__ void put(int q, float4 h, float4 l)
    {
        const int p = q >> 1, o = q & 1;
        float* A = reinterpret_cast<float*>(&a[p]) + o;
        float* B = reinterpret_cast<float*>(&b[p]) + o;
        float* C = reinterpret_cast<float*>(&c[p]) + o;
        float* D = reinterpret_cast<float*>(&d[p]) + o;
        A[0] = h.x; A[2] = h.y; B[0] = l.x; B[2] = l.y;
        C[0] = h.z; C[2] = l.z; D[0] = h.w; D[2] = l.w;
    }
    // source 2p (odd = 0) or 2p + 1 as (x, y, z, m) hi and lo
    __device__ __forceinline__ void get(int p, int odd, float4& h, float4& l) const
    {
        const float4 A = a[p], B = b[p], C = c[p], D = d[p];
        h = odd ? make_float4(A.y, A.w, C.y, D.y) : make_float4(A.x, A.z, C.x, D.x);
        l = odd ? make_float4(B.y, B.w, C.w, D.w) : make_float4(B.x, B.z, C.z, D.z);
    }
};

// For sums of at most np terms.  False: the leaf is not distant (max R over
// min R may exceed kFarRatio, or min R < r_floor).
template <int DIM>
__device__ __forceinline__ bool far_setup(const float* T, const LeafBox& box, int np, float e2h,
                                          float e2l, float r_floor, FarLeaf& f)
{
    float g[3] = {0.f, 0.f, 0.f}, rmin = e2h, rmax = e2h;
#pragma unroll
    for (int k = 0; k < DIM; k++) {
        g[k] = __fsub_rn(comp(box.c, k), T[k]);
        const float h = comp(box.h, k);
        const float near = fmaxf(fabsf(g[k]) - h, 0.0f), away = fabsf(g[k]) + h;
        rmin = fmaf(near, near, rmin);
        rmax = fmaf(away, away, rmax);
    }
    rmax *= 1.0f + 0x1p-20f;
    f.s0 = rmax;
    f.si = __fadd_rn(rmax, e2h);
    f.li = __fadd_rn(__fsub_rn(e2h, __fsub_rn(f.si, rmax)), e2l);
    // |term k| <= 1.84 |m| |d_k| / rmin^(3/2), |d_k| <= away_k; terms of the
    // other sign only where the target is inside the box's slab, and then
    // |d_k| <= h_k - |g_k| (any |d_k| with masses of both signs)
    const float ri = rsqrt_mufu(fmaxf(rmin, 0x1p-80f));
    const float u = 3.69f * fabsf(box.c.w) * (ri * ri * ri);
    const float n = (float)np;
#pragma unroll
    for (int k = 0; k < DIM; k++) {
        const float ak = fabsf(g[k]), h = comp(box.h, k);
        const float take = box.c.w < 0.0f ? ak + h : fmaxf(h - ak, 0.0f);
        const float B = u * fmaf(n, take, ak + h);
        f.b[k] = copysignf(
            __int_as_float((__float_as_int(B) & 0x7f800000) + 0x00800000), g[k]);
    }
    return rmin * kFarRatio >= rmax && rmin >= r_floor;
}

static __device__ __forceinline__ float2 both(float v) { return make_float2(v, v); }

// -v by the sign bits: two ALU instructions, where the FP32 pipe is the
// scarce one.
static __device__ __forceinline__ float2 neg2(float2 v)
{
    return make_float2(__int_as_float(__float_as_int(v.x) ^ 0x80000000),
                       __int_as_float(__float_as_int(v.y) ^ 0x80000000));
}

// -v / 2 of positive normal numbers above 2^-125, by one ALU addition each.
static __device__ __forceinline__ float2 neg_half2(float2 v)
{
    return make_float2(__int_as_float(__float_as_int(v.x) + 0x7f800000),
                       __int_as_float(__float_as_int(v.y) + 0x7f800000));
}

// Rows p = sub, sub + step, ... of a staged distant leaf of cn sources, as an
// unbiased float-float sum.
template <int DIM, bool UNIT>
__device__ __forceinline__ void far_pairs(const float* Th, const float* Tl, const LeafStage& st,
                                          int sub, int step, int cn, const FarLeaf& f, float* ph,
                                          float* pl)
{
    float2 ah[3], al[3], nT[3], nL[3];
#pragma unroll
    for (int k = 0; k < DIM; k++) {
        ah[k] = both(f.b[k]);
        al[k] = both(0.0f);
        nT[k] = both(-Th[k]);
        nL[k] = both(-Tl[k]);
    }
    const float2 m1 = both(-1.0f), two = both(2.0f);
    const int np = (cn + 1) >> 1;
    // from the last row down: its odd source may not exist (a lane beyond the
    // rows has none)
#pragma unroll 1
    for (int p = sub < np ? sub + (np - 1 - sub) / step * step : -1; p >= 0; p -= step) {
        const float4 A = st.a[p], B = st.b[p];
        float4 C = make_float4(0.f, 0.f, 0.f, 0.f);
        if (DIM == 3) C = st.c[p];
        const float2 xh[3] = {make_float2(A.x, A.y), make_float2(A.z, A.w), make_float2(C.x, C.y)};
        const float2 xl[3] = {make_float2(B.x, B.y), make_float2(B.z, B.w), make_float2(C.z, C.w)};
        float2 d[3], l[3], s = both(f.si), lo = both(f.li);
#pragma unroll
        for (int k = 0; k < DIM; k++) {
            d[k] = __fadd2_rn(xh[k], nT[k]);              // exact on the grid
            l[k] = __fadd2_rn(xl[k], nL[k]);
            const float2 t = __ffma2_rn(d[k], d[k], s);
            const float2 q = __ffma2_rn(d[k], d[k], __ffma2_rn(t, m1, s));
            lo = __ffma2_rn(__ffma2_rn(two, d[k], l[k]), l[k], lo);
            lo = __fadd2_rn(lo, q);
            s = t;
        }
        const float2 R0 = __fadd2_rn(s, both(-f.s0));     // exact: s <= 2 s0
        const float2 rs = __ffma2_rn(lo, both(2.0f / 3.0f), __fmul2_rn(R0, both(2.0f / 3.0f)));
        const float2 y = make_float2(rsqrt_mufu(rs.x), rsqrt_mufu(rs.y));
        const float2 Y = __fmul2_rn(y, y);
        const float2 Ye = __ffma2_rn(y, y, neg2(Y));
        const float2 A1 = __ffma2_rn(lo, Y, __ffma2_rn(R0, Y, both(-1.5f)));
        const float2 W = __fmul2_rn(Y, y), nW = neg2(W);
        const float2 We = __ffma2_rn(Ye, neg_half2(y), __ffma2_rn(Y, y, nW));
        float2 fh = W, fl = __ffma2_rn(nW, A1, We);
        if (!UNIT) {
            const float4 M = st.d[p];
            const float2 mh = make_float2(M.x, M.y), ml = make_float2(M.z, M.w);
            fh = __fmul2_rn(mh, W);
            fl = __ffma2_rn(mh, fl, __ffma2_rn(ml, W, __ffma2_rn(mh, W, neg2(fh))));
        }
#pragma unroll
        for (int k = 0; k < DIM; k++) {
            const float2 t = __ffma2_rn(fh, d[k], ah[k]);
            float2 r = __ffma2_rn(fh, d[k], __ffma2_rn(t, m1, ah[k]));
            r = __ffma2_rn(fl, d[k], r);
            r = __ffma2_rn(fh, l[k], r);
            al[k] = __fadd2_rn(al[k], r);
            ah[k] = t;
        }
        if (2 * p + 1 >= cn) {   // no odd source (this lane's first row): start over
#pragma unroll
            for (int k = 0; k < DIM; k++) { ah[k].y = f.b[k]; al[k].y = 0.0f; }
        }
    }
#pragma unroll
    for (int k = 0; k < DIM; k++) {
        const float hx = __fsub_rn(ah[k].x, f.b[k]), hy = __fsub_rn(ah[k].y, f.b[k]);
        const float h = __fadd_rn(hx, hy);
        const float l = __fadd_rn(two_sum_err(hx, hy, h), __fadd_rn(al[k].x, al[k].y));
        ph[k] = __fmul_rn(h, kFarScale);
        pl[k] = __fmaf_rn(l, kFarScale, __fmaf_rn(h, kFarScaleLo, __fmaf_rn(h, kFarScale, -ph[k])));
    }
}

// The same rows of a near leaf with pair_ff_soft, added to (ph, pl).
template <int DIM, bool UNIT>
__device__ __forceinline__ void near_pairs(const float* Th, const float* Tl, const LeafStage& st,
                                           int sub, int step, int cn, float e2h, float e2l,
                                           float* ph, float* pl)
{
#pragma unroll 1
    for (int p = sub; 2 * p < cn; p += step) {
        float4 h, l;
        st.get(p, 0, h, l);
        pair_ff_soft<DIM, UNIT>(Th, Tl, h, l, e2h, e2l, ph, pl);
        if (2 * p + 1 < cn) {
            st.get(p, 1, h, l);
            pair_ff_soft<DIM, UNIT>(Th, Tl, h, l, e2h, e2l, ph, pl);
        }
    }
}

// Lanes of a leaf visit.  More than kSplitMaxK active targets: every lane
// works for itself.  Fewer, k: f lanes for each active target; lane j works
// for the active target of rank j / f.
struct LaneSplit {
    int f = 1, sub = 0, owner, leader;
    bool work;
    __device__ __forceinline__ LaneSplit(unsigned mask, int lane)
    {
        const int k = __popc(mask);
        owner = leader = lane;
        work = (mask >> lane) & 1u;
        if (k <= kSplitMaxK) {
            const bool mine = work;
            f = 2;
            while (f * 2 * k <= kWarp) f *= 2;
            const int r = lane / f;
            sub = lane & (f - 1);
            work = r < k;
            owner = nth_set_bit(mask, work ? r : 0);
            leader = mine ? __popc(mask & ((1u << lane) - 1u)) * f : 0;
        }
    }
};

// The lanes' partial sums (ph, pl) of a visit, added in a fixed order per
// target and to the accumulators (ah, al) of the active lanes.
template <int DIM>
__device__ __forceinline__ void split_add(const LaneSplit& sp, bool mine, float* ph, float* pl,
                                          float* ah, float* al)
{
    const unsigned FULL = 0xffffffffu;
    if (sp.f > 1) {
        for (int o = sp.f >> 1; o >= 1; o >>= 1) {
#pragma unroll
            for (int c = 0; c < DIM; c++) {
                const float bh = __shfl_down_sync(FULL, ph[c], o);
                const float bl = __shfl_down_sync(FULL, pl[c], o);
                ff_add(ph[c], pl[c], bh, bl);
            }
        }
#pragma unroll
        for (int c = 0; c < DIM; c++) {
            ph[c] = __shfl_sync(FULL, ph[c], sp.leader);
            pl[c] = __shfl_sync(FULL, pl[c], sp.leader);
        }
    }
    if (mine) {
#pragma unroll
        for (int c = 0; c < DIM; c++) ff_add(ah[c], al[c], ph[c], pl[c]);
    }
}

// The coordinates a lane works on in a visit: its own target's, or those of
// the target it was given.
template <int DIM>
__device__ __forceinline__ void split_target(const LaneSplit& sp, const float* Th, const float* Tl,
                                             float* T, float* L)
{
#pragma unroll
    for (int c = 0; c < DIM; c++) {
        T[c] = Th[c];
        L[c] = Tl[c];
        if (sp.f > 1) {
            T[c] = __shfl_sync(0xffffffffu, Th[c], sp.owner);
            L[c] = __shfl_sync(0xffffffffu, Tl[c], sp.owner);
        }
    }
}

// One staged block of cn <= kStage leaf particles for the targets of the lanes in
// `mask` (those that opened the leaf's parent), float-float soft path
// (far_pairs when the leaf is distant for every working lane, else
// pair_ff_soft).  Called by all 32 lanes.
//
// With more than 16 active lanes each lane sums its own target's pairs.  With
// k <= 16 active lanes the idle lanes are put to work: every active target
// gets f lanes (f = 2..32, the largest power of two with f k <= 32); lane j
// works for the active target of rank j / f, on the rows (two sources)
// j mod f, j mod f + f, ..., into a float-float partial sum; the f partials
// are added in a fixed tree order (shuffles down by f/2, f/4, ..., 1) and the
// sum is added to the target's accumulator with ff_add.  Leaf visits with at
// most 16 active lanes carry most of the warp's idle lanes (a CPU replay of
// the walk at 1M Plummer, theta 0.5, leaf 32: 16 % of the leaf steps, 84 % of
// the idle lane-steps), and the split cuts the pair steps of a solve by about
// a tenth.  The order of every addition depends only on the mask and cn, so a
// result does not depend on which kernel (single tree or batched) evaluates
// it.  One loop serves full and split visits: the loops' code competes for
// the instruction cache.
template <int DIM, bool UNIT>
__device__ __forceinline__ void leaf_block_soft(unsigned mask, int lane, const float* Th,
                                                const float* Tl, const LeafStage& st, int cn,
                                                const LeafBox& box, float e2h, float e2l,
                                                float* ah, float* al)
{
    const unsigned FULL = 0xffffffffu;
    if (mask == 0) return;
    const LaneSplit sp(mask, lane);
    float T[3] = {0.f, 0.f, 0.f}, L[3] = {0.f, 0.f, 0.f};
    split_target<DIM>(sp, Th, Tl, T, L);
    float ph[3] = {0.f, 0.f, 0.f}, pl[3] = {0.f, 0.f, 0.f};
    FarLeaf f;
    const bool far = far_setup<DIM>(T, box, (cn + 1) >> 1, e2h, e2l, 0.0f, f);
    if (__all_sync(FULL, far || !sp.work)) {
        if (sp.work) far_pairs<DIM, UNIT>(T, L, st, sp.sub, sp.f, cn, f, ph, pl);
    } else {
        if (sp.work) near_pairs<DIM, UNIT>(T, L, st, sp.sub, sp.f, cn, e2h, e2l, ph, pl);
    }
    split_add<DIM>(sp, (mask >> lane) & 1u, ph, pl, ah, al);
}

// The LeafBox of particles [start, start + count).
static __device__ __forceinline__ void leaf_box(const float4* __restrict__ ph, int start,
                                                int count, float4& c, float4& h)
{
    float lo[3] = {4.f, 4.f, 4.f}, hi[3] = {-4.f, -4.f, -4.f}, mx = 0.0f;
    bool neg = false;
#pragma unroll 8
    for (int i = start; i < start + count; i++) {
        const float4 p = ph[i];
#pragma unroll
        for (int k = 0; k < 3; k++) {
            lo[k] = fminf(lo[k], comp(p, k));
            hi[k] = fmaxf(hi[k], comp(p, k));
        }
        mx = fmaxf(mx, fabsf(p.w));
        neg |= p.w < 0.0f;
    }
    c = make_float4(0.5f * (lo[0] + hi[0]), 0.5f * (lo[1] + hi[1]), 0.5f * (lo[2] + hi[2]),
                    neg ? -mx : mx);
    const float s = 1.0f + 0x1p-20f, o = 0x1p-21f;
    h = make_float4(fmaf(0.5f * (hi[0] - lo[0]), s, o), fmaf(0.5f * (hi[1] - lo[1]), s, o),
                    fmaf(0.5f * (hi[2] - lo[2]), s, o), 0.0f);
}

// Header of a node, one load per visit: leaf (-1, start, count, flag), any node
// without mass (-1, start, 0, 0); internal (first child, size, |com - box
// centre| as float bits, flag).  Flags: see node_flag; kTwig and the counts at
// bits 8 and 16 for a twig, an internal node whose children are leaves of
// neighbouring particles (at most 32 each, with mass): a target that opens it
// takes both leaves, which need no visit of their own.
constexpr int kNodeMass = 1, kNodeOutside = 2, kTwig = 4;
static __device__ __forceinline__ int twig_left(int w) { return (w >> 8) & 0xff; }
static __device__ __forceinline__ int twig_right(int w) { return (w >> 16) & 0xff; }

// What the traversals read of node k (FP32 copies in frame f), from the tree
// and the particles' copies ph.
static __device__ __forceinline__ void put_node(const TreeDev& t, int64_t k, const FastFrame& f,
                                                bool fine, const double* __restrict__ center,
                                                const double* __restrict__ quad,
                                                const float4* __restrict__ ph, const NodeCopies& o)
{
    const NodeCM c = t.cm[k];
    const int dim = t.dim, fc = t.first_child[k];
    float4 h, l;
    split_grid(c.x, f.c[0], f.s, fine, h.x, l.x);
    split_grid(c.y, f.c[1], f.s, fine, h.y, l.y);
    if (dim == 3) split_grid(c.z, f.c[2], f.s, fine, h.z, l.z);
    else h.z = l.z = 0.0f;
    split_plain(__dmul_rn(c.w, f.ms), h.w, l.w);
    int4 hd;
    if (fc < 0) {
        // (a LeafBox in a leaf's place; form "fp32" reads neither)
        if (fine) leaf_box(ph, t.start[k], t.count[k], h, l);
        hd = make_int4(fc, t.start[k], t.count[k], c.w != 0.0 ? kNodeMass : 0);
    } else {
        // distance between the centre of mass and the AABB centre (offset MAC)
        double dd = 0.0;
        for (int d = 0; d < dim; d++) {
            const double cc = d == 0 ? c.x : (d == 1 ? c.y : c.z);
            const double v = cc - center[k * dim + d];
            dd += v * v;
        }
        int flag = node_flag(c, h);
        if (flag && t.first_child[fc] < 0 && t.first_child[fc + 1] < 0) {
            const int s = t.start[fc], n0 = t.count[fc], n1 = t.count[fc + 1];
            if (n0 >= 1 && n1 >= 1 && n0 <= kWarp && n1 <= kWarp && t.start[fc + 1] == s + n0 &&
                t.cm[fc].w != 0.0 && t.cm[fc + 1].w != 0.0) {
                flag |= kTwig | n0 << 8 | n1 << 16;
                if (o.twig) {
                    LeafBox b;
                    leaf_box(ph, s, n0 + n1, b.c, b.h);
                    b.h.w = __int_as_float(s);
                    o.twig[k] = b;
                }
            }
        }
        hd = make_int4(fc, __float_as_int(__double2float_rn(__dmul_rn(t.size[k], f.s))),
                       __float_as_int(__double2float_ru(sqrt(dd) * f.s)), flag);
    }
    if (!hd.w) hd = make_int4(-1, t.start[k], 0, 0);   // without mass: skipped (bh.py:514)
    o.nh[k] = h;
    o.nl[k] = l;
    o.nhdr[k] = hd;
    if (quad) {   // mass x length^2: scale by ms s^2
        const double qs = f.ms * f.s * f.s;
        const double* q = quad + 6 * k;
        o.nq0[k] = make_float4((float)(q[0] * qs), (float)(q[1] * qs), (float)(q[2] * qs),
                               (float)(q[3] * qs));
        o.nq1[k] = make_float2((float)(q[4] * qs), (float)(q[5] * qs));
    }
}

// FP64 pair in physical units, G-less (the Numba loop arithmetic).
template <int DIM>
__device__ __forceinline__ void pair_fp64(double x, double y, double z, double px, double py,
                                          double pz, double pm, double eps2, double* a64)
{
    const double dx = __dsub_rn(px, x), dy = __dsub_rn(py, y);
    const double dz = DIM == 3 ? __dsub_rn(pz, z) : 0.0;
    double r2 = __dmul_rn(dx, dx);
    r2 = __dadd_rn(r2, __dmul_rn(dy, dy));
    if (DIM == 3) r2 = __dadd_rn(r2, __dmul_rn(dz, dz));
    r2 = __dadd_rn(r2, eps2);
    if (r2 == 0.0) return;
    const double ri = __ddiv_rn(1.0, __dsqrt_rn(r2));
    const double f = __dmul_rn(pm, __dmul_rn(__dmul_rn(ri, ri), ri));
    a64[0] = __dadd_rn(a64[0], __dmul_rn(f, dx));
    a64[1] = __dadd_rn(a64[1], __dmul_rn(f, dy));
    if (DIM == 3) a64[2] = __dadd_rn(a64[2], __dmul_rn(f, dz));
}

// Exact opening test (bh.py:576-601), same arithmetic as k_traverse_exact.
template <int DIM>
__device__ __forceinline__ bool open_exact64(double x, double y, double z, const NodeCM& cm,
                                             double size, double theta)
{
    double dx = __dsub_rn(x, cm.x), dy = __dsub_rn(y, cm.y);
    double s;
    if (DIM == 3) {
        double dz = __dsub_rn(z, cm.z);
        s = __fma_rn(dz, dz, __fma_rn(dy, dy, __dmul_rn(dx, dx)));
    } else {
        s = __fma_rn(dy, dy, __dmul_rn(dx, dx));
    }
    double d = __dsqrt_rn(s);
    if (d == 0.0) return true;
    return __ddiv_rn(size, d) >= theta;
}


// Displacement from the hi parts (exact on the grid) plus the lo parts
// (exact on their grid), rounded once: FP32-relative accuracy everywhere in
// the box, also in dense regions far from the box centre.
template <int DIM>
__device__ __forceinline__ void pair_f32(const float* Th, const float* Tl, float4 sh, float4 sl,
                                         float e2, float* acc, float* cmp)
{
    const float d0 = __fadd_rn(__fsub_rn(sh.x, Th[0]), __fsub_rn(sl.x, Tl[0]));
    const float d1 = __fadd_rn(__fsub_rn(sh.y, Th[1]), __fsub_rn(sl.y, Tl[1]));
    const float d2 = DIM == 3 ? __fadd_rn(__fsub_rn(sh.z, Th[2]), __fsub_rn(sl.z, Tl[2])) : 0.0f;
    float r2 = fmaf(d1, d1, fmaf(d0, d0, e2));
    if (DIM == 3) r2 = fmaf(d2, d2, r2);
    // r^2 + eps^2 == 0: no force (kernels.py:62-63); below the normal range
    // (closer than 2^-63 box sizes, unsoftened) the FP32 force would
    // overflow: none either.  Selected, not branched: f = 0 then.
    const bool ok = r2 >= 0x1p-126f;
    const float ri = rsqrt_mufu(ok ? r2 : 1.0f);
    const float f = ok ? sh.w * (ri * ri * ri) : 0.0f;
    const float d[3] = {d0, d1, d2};
#pragma unroll
    for (int k = 0; k < DIM; k++) {            // Kahan compensated sum
        const float y = fmaf(f, d[k], -cmp[k]);
        const float t = __fadd_rn(acc[k], y);
        cmp[k] = __fsub_rn(__fsub_rn(t, acc[k]), y);
        acc[k] = t;
    }
}


// A target's negated hi and lo coordinates, x and y packed for the f32x2
// instructions of pair_f32_partial2.
struct TargetF32x2 {
    float2 hxy, lxy;
    float hz, lz;
};

static __device__ __forceinline__ TargetF32x2 target_f32x2(const float* T, const float* Tl)
{
    TargetF32x2 t;
    t.hxy = make_float2(-T[0], -T[1]);
    t.lxy = make_float2(-Tl[0], -Tl[1]);
    t.hz = -T[2];
    t.lz = -Tl[2];
    return t;
}

// FP32 pair term added to a plain FP32 partial sum (pxy, pz): the leaf loop
// sums at most 32 such terms and then adds the partial to the Kahan-compensated
// per-target accumulator with kahan_add_f32 (blocked Kahan summation).  Same
// displacement, r^2 and force as pair_f32, with the x and y components in
// Blackwell's f32x2 instructions (FADD2 / FFMA2: two IEEE single operations per
// issue slot; x - y is x + (-y) exactly).  CHECK = false: the caller guarantees
// e2 >= 2^-126; r^2 is an FMA chain of non-negative terms started at e2, so
// r^2 >= e2 and the test is compiled out.  UNIT: the source's mass is exactly 1
// (the unit-mass frame) and the product with it is skipped, also exactly.
template <int DIM, bool CHECK, bool UNIT>
__device__ __forceinline__ void pair_f32_partial2(const TargetF32x2& t, float4 sh, float4 sl,
                                                  float e2, float2& pxy, float& pz)
{
    const float2 dxy = __fadd2_rn(__fadd2_rn(make_float2(sh.x, sh.y), t.hxy),
                                  __fadd2_rn(make_float2(sl.x, sl.y), t.lxy));
    const float dz = DIM == 3 ? __fadd_rn(__fadd_rn(sh.z, t.hz), __fadd_rn(sl.z, t.lz)) : 0.0f;
    float r2 = fmaf(dxy.y, dxy.y, fmaf(dxy.x, dxy.x, e2));
    if (DIM == 3) r2 = fmaf(dz, dz, r2);
    const bool ok = !CHECK || r2 >= 0x1p-126f;
    const float ri = rsqrt_mufu(ok ? r2 : 1.0f);
    const float w = ri * ri * ri;
    const float f = ok ? (UNIT ? w : sh.w * w) : 0.0f;
    pxy = __ffma2_rn(make_float2(f, f), dxy, pxy);
    if (DIM == 3) pz = fmaf(f, dz, pz);
}

// Rows first .. first + np - 1 of a staged block (two sources to a row) for a
// target with negated coordinates (nT, nL): displacements, r^2 and w = r^-3 of both
// sources in f32x2 instructions, the forces added to the partial sum p one
// source after the other.  Every operation and its order are those of
// pair_f32_partial2, so the sums are the same bit for bit.  UNIT: masses are
// exactly 1 and their products are skipped, also exactly.  np is even; places
// past the last source hold stand-ins that add exactly zero.  (In steps of four
// rows, leaves of 33 to 64 particles took up to 1.22 times as long as one source
// at a time, for the stand-ins and registers spilled: 300k galaxy in leaves of 48
// 20.7 ms, by two rows 20.0, one by one 19.5; 256 systems in leaves of 16 41.8,
// 39.8 and, without leaf pairs, 56.8.)
template <int DIM, bool CHECK, bool UNIT>
__device__ __forceinline__ void rows_f32(const LeafStage& st, int first, int np, const float2* nT,
                                         const float2* nL, float e2, float* p)
{
    for (int r0 = first; r0 < first + np; r0 += 2)
#pragma unroll
    for (int r = r0; r < r0 + 2; r++) {
        const float4 A = st.a[r], B = st.b[r];
        const float2 dx = __fadd2_rn(__fadd2_rn(make_float2(A.x, A.y), nT[0]),
                                     __fadd2_rn(make_float2(B.x, B.y), nL[0]));
        const float2 dy = __fadd2_rn(__fadd2_rn(make_float2(A.z, A.w), nT[1]),
                                     __fadd2_rn(make_float2(B.z, B.w), nL[1]));
        float2 dz = both(0.0f), r2 = __ffma2_rn(dy, dy, __ffma2_rn(dx, dx, both(e2)));
        if (DIM == 3) {
            const float4 C = st.c[r];
            dz = __fadd2_rn(__fadd2_rn(make_float2(C.x, C.y), nT[2]),
                            __fadd2_rn(make_float2(C.z, C.w), nL[2]));
            r2 = __ffma2_rn(dz, dz, r2);
        }
        const bool ok0 = !CHECK || r2.x >= 0x1p-126f, ok1 = !CHECK || r2.y >= 0x1p-126f;
        const float2 ri = make_float2(rsqrt_mufu(ok0 ? r2.x : 1.0f), rsqrt_mufu(ok1 ? r2.y : 1.0f));
        float2 f = __fmul2_rn(__fmul2_rn(ri, ri), ri);
        if (!UNIT) {
            const float4 M = st.d[r];
            f = __fmul2_rn(make_float2(M.x, M.y), f);
        }
        if (CHECK) f = make_float2(ok0 ? f.x : 0.0f, ok1 ? f.y : 0.0f);
        p[0] = fmaf(f.x, dx.x, p[0]);
        p[1] = fmaf(f.x, dy.x, p[1]);
        if (DIM == 3) p[2] = fmaf(f.x, dz.x, p[2]);
        p[0] = fmaf(f.y, dx.y, p[0]);
        p[1] = fmaf(f.y, dy.y, p[1]);
        if (DIM == 3) p[2] = fmaf(f.y, dz.y, p[2]);
    }
}


// Rows that rows_f32 takes for c sources.
static __device__ __forceinline__ int rows_for(int c) { return ((c + 3) >> 2) << 1; }

// Stages two runs of at most 32 sources for rows_f32, the second (which may be
// empty) in the rows after the first's.  Stand-ins fill the rows: for targets
// in the box (|T| <= 1) far away, so that r^2 is about 3e36 and r^-3 rounds to
// zero; when some target lies outside, without mass (the masses must then be
// used), at a point off every grid.
static __device__ __forceinline__ void stage_f32(LeafStage& st, int lane, const float4* ph,
                                                 const float4* pl, int s0, int c0, int s1, int c1,
                                                 bool outside)
{
    const int n0 = 2 * rows_for(c0), n = n0 + 2 * rows_for(c1);
    const float v = outside ? 3.14159265f : 1e18f;
    for (int j = lane; j < n; j += kWarp) {
        const int q = j < n0 ? j : j - n0;
        float4 h = make_float4(v, v * 1.25f, v * 1.5f, 0.0f), l = make_float4(0.f, 0.f, 0.f, 0.f);
        if (q < (j < n0 ? c0 : c1)) {
            const int at = (j < n0 ? s0 : s1) + q;
            h = ph[at];
            l = pl[at];
        }
        st.put(j, h, l);
    }
}

template <int DIM>
__device__ __forceinline__ void kahan_add_f32(const float* p, float* acc, float* cmp)
{
#pragma unroll
    for (int k = 0; k < DIM; k++) {
        const float y = __fsub_rn(p[k], cmp[k]);
        const float t = __fadd_rn(acc[k], y);
        cmp[k] = __fsub_rn(__fsub_rn(t, acc[k]), y);
        acc[k] = t;
    }
}

// Opening test of the FP32 form, on the hi coordinates (exact differences on
// the 2^-23 grid).  The criterion is a heuristic, so a decision at the margin
// may go either way, but always the same way: `opens` is the definition, and
// the squares, which need no square root, decide where they are further apart
// than both forms' rounding (2^-18 of them; each is a handful of roundings).
// mac 1: the offset criterion, open when d < size / theta + |com - centre|.
struct OpenF32 {
    float theta, inv, mac;   // mac: 1 or 0, the weight of |com - centre|
    __device__ __forceinline__ OpenF32(double th, int m)
        : theta((float)th), inv(1.0f / (float)th), mac(m == 1 ? 1.0f : 0.0f) {}
    __device__ __forceinline__ bool opens(float d2, float size, float off) const
    {
        const float dist = d2 > 0.0f ? d2 * rsqrtf(d2) : 0.0f;
        if (mac != 0.0f) return size >= theta * (dist - off);
        return dist == 0.0f || size >= theta * dist;
    }
    // squares outside the band decide, the root inside it (lanes outside `act`
    // return anything); two nodes share the rare branch
    __device__ __forceinline__ bool near(float d2, float size, float off, bool& open) const
    {
        const float r = fmaf(off, mac, size * inv), r2 = r * fabsf(r);   // (negative: never opens)
        open = r2 >= d2;
        return !(fabsf(r2 - d2) > 0x1p-18f * d2);
    }
    __device__ __forceinline__ bool operator()(float d2, float size, float off, bool act) const
    {
        bool open;
        if (near(d2, size, off, open) && act) open = opens(d2, size, off);
        return open;
    }
};

// A node's monopole plus its Plummer-softened traceless quadrupole (FP32
// form, multipole "quad"), Kahan-added.  With d = com - x (target to node),
// r^2 = |d|^2 + eps^2:
//   a = M d / r^3 - Q d / r^5 + (5/2) (d . Q d) d / r^7,
// the gradient of the potential -M/r - (1/2) d.Q d / r^5.
template <int DIM>
__device__ __forceinline__ void node_quad_f32(const float* Th, const float* Tl, float4 nh,
                                              float4 nl, float4 q0, float2 q1, float e2,
                                              float* acc, float* cmp)
{
    const float d0 = __fadd_rn(__fsub_rn(nh.x, Th[0]), __fsub_rn(nl.x, Tl[0]));
    const float d1 = __fadd_rn(__fsub_rn(nh.y, Th[1]), __fsub_rn(nl.y, Tl[1]));
    const float d2 = DIM == 3 ? __fadd_rn(__fsub_rn(nh.z, Th[2]), __fsub_rn(nl.z, Tl[2])) : 0.0f;
    float r2 = fmaf(d1, d1, fmaf(d0, d0, e2));
    if (DIM == 3) r2 = fmaf(d2, d2, r2);
    if (!(r2 >= 0x1p-126f)) return;
    const float ri = rsqrt_mufu(r2);
    const float ri2 = ri * ri;
    const float ri3 = ri2 * ri;
    const float ri5 = ri3 * ri2;
    const float qx = fmaf(q1.x, d2, fmaf(q0.w, d1, q0.x * d0));
    const float qy = fmaf(q1.y, d2, fmaf(q0.y, d1, q0.w * d0));
    const float qz = fmaf(q0.z, d2, fmaf(q1.y, d1, q1.x * d0));
    const float dqd = fmaf(d2, qz, fmaf(d1, qy, d0 * qx));
    const float f = fmaf(2.5f * dqd, ri5 * ri2, nh.w * ri3);
    const float d[3] = {d0, d1, d2}, q[3] = {qx, qy, qz};
#pragma unroll
    for (int k = 0; k < DIM; k++) {
        const float y = __fsub_rn(fmaf(f, d[k], -ri5 * q[k]), cmp[k]);
        const float t = __fadd_rn(acc[k], y);
        cmp[k] = __fsub_rn(__fsub_rn(t, acc[k]), y);
        acc[k] = t;
    }
}

// The warp's traversal stack (left children; the right child of an opened node
// is visited next) of (node, lanes, lanes that open it) entries, two placements:
//  STK 0: in shared memory, lane 0 writes, every lane reads (__syncwarp
//         around each pop);
//  STK 1: in registers, entry j held by lane j % 32 in register j / 32;
//         a pop is three shuffles from the owning lane, a push a predicated
//         register write; no shared memory, no __syncwarp.
// Entries are warp-uniform, so every lane keeps the same depth `sp`.
struct StackEntry {
    int node;
    unsigned mask, open;
};
template <int STK> struct WarpStack;

template <> struct WarpStack<0> {
    StackEntry* s;
    int sp = 0, lane;
    __device__ WarpStack(StackEntry* s_, int lane_) : s(s_), lane(lane_) {}
    __device__ StackEntry pop()
    {
        __syncwarp();
        const StackEntry e = s[--sp];
        __syncwarp();
        return e;
    }
    __device__ void push(const StackEntry& e)
    {
        if (lane == 0) s[sp] = e;
        sp++;
    }
};

template <> struct WarpStack<1> {
    static_assert(kStackDepth <= 2 * kWarp, "register stack holds two entries per lane");
    StackEntry e0{0, 0, 0}, e1{0, 0, 0};
    int sp = 0, lane;
    __device__ WarpStack(StackEntry*, int lane_) : lane(lane_) {}
    __device__ StackEntry pop()
    {
        --sp;
        const bool hi = sp >= kWarp;
        return {__shfl_sync(0xffffffffu, hi ? e1.node : e0.node, sp & 31),
                __shfl_sync(0xffffffffu, hi ? e1.mask : e0.mask, sp & 31),
                __shfl_sync(0xffffffffu, hi ? e1.open : e0.open, sp & 31)};
    }
    __device__ void push(const StackEntry& e)
    {
        if (lane == (sp & 31)) {
            if (sp < kWarp) e0 = e;
            else e1 = e;
        }
        sp++;
    }
};

// FP32 walk of a warp's targets (negated coordinates nT, nL for the rows) from
// node `root`, shared by the single trees (FastTree) and the batches.  The
// children of an opened node are tested together, so a node costs half a test
// and half the loop around it; its left child waits in registers and goes to
// the stack only when the right one is opened too.  Contributions reach a
// target in the order of a walk that visits right before left.  The kernels
// issue on 79 % of the clocks, so what counts is instructions: 2M galaxy, theta
// 0.7, leaf 16, node by node 106.6 ms, by pairs 103.3, with one branch for both
// roots and no separate test for mass 101.2 (1M of it: 38.5 G warp
// instructions; rows about 12, monopoles 6, visits 19).  Separate kernels with
// and without the small-r test: 100.9, batches 42.5 against 42.2, not kept.
template <int DIM, class TREE, class STACK>
__device__ __forceinline__ void walk_f32(const TREE& ft, int root, int lane, bool valid, int me,
                                         bool outside, bool unit, const OpenF32& opener, float e2h,
                                         const float* T, const float* Tl, float* acc, float* cmp,
                                         STACK& st, LeafStage& stage, unsigned* cnt,
                                         bool& overflow)
{
    const unsigned FULL = 0xffffffffu;
    const bool soft = e2h >= 0x1p-126f;   // r^2 >= eps^2 is normal: no small-r test
    const float2 nT[3] = {both(-T[0]), both(-T[1]), both(-T[2])};
    const float2 nL[3] = {both(-Tl[0]), both(-Tl[1]), both(-Tl[2])};
    const auto dist2 = [&](const float4& nh) {
        float d2 = 0.0f;
#pragma unroll
        for (int k = 0; k < DIM; k++) {
            const float d = __fsub_rn(comp(nh, k), T[k]);
            d2 = fmaf(d, d, d2);
        }
        return d2;
    };
    StackEntry e{root, __ballot_sync(FULL, valid), 0};   // the node, lanes that reach and open it
    StackEntry left{-1, 0, 0};                           // the sibling that comes next
    int4 hd = ft.nhdr[root];                             // (first_child, start, count, flag)
    e.open = __ballot_sync(FULL, opener(dist2(ft.nh[root]), __int_as_float(hd.y),
                                        __int_as_float(hd.z), valid) && valid);
    cnt[2] += valid;
    while (true) {
        // runs of particles to take: a leaf's blocks of 32, or a twig's right
        // and left leaf (the order in which the leaves would be visited)
        unsigned lmask = 0;
        int s0 = hd.y, c0 = 0, s1 = 0, c1 = 0;
        const int fc = hd.x;
        if (fc < 0) {                     // (without mass: no particles, put_node)
            lmask = e.mask;
            c0 = hd.z;
        } else {
            if (((e.mask & ~e.open) >> lane) & 1u) {
                if (ft.nq0)
                    node_quad_f32<DIM>(T, Tl, ft.nh[e.node], ft.nl[e.node], ft.nq0[e.node],
                                       ft.nq1[e.node], e2h, acc, cmp);
                else
                    pair_f32<DIM>(T, Tl, ft.nh[e.node], ft.nl[e.node], e2h, acc, cmp);
                cnt[1]++;
            }
            if (e.open && (hd.w & kTwig)) {
                lmask = e.open;
                s1 = ft.nhdr[fc].y;
                c1 = twig_left(hd.w);
                s0 = s1 + c1;
                c0 = twig_right(hd.w);
                cnt[2] += (lmask >> lane) & 1u ? 2 : 0;
            } else if (e.open) {
                if (left.node >= 0) {
                    if (st.sp + 3 > kStackDepth) { overflow = true; break; }
                    st.push(left);
                }
                const int4 hl = ft.nhdr[fc];
                hd = ft.nhdr[fc + 1];
                const float dl = dist2(ft.nh[fc]), dr = dist2(ft.nh[fc + 1]);
                const bool act = (e.open >> lane) & 1u;
                cnt[2] += act ? 2 : 0;
                bool ol, orr;
                const bool nl = opener.near(dl, __int_as_float(hl.y), __int_as_float(hl.z), ol);
                const bool nr = opener.near(dr, __int_as_float(hd.y), __int_as_float(hd.z), orr);
                if (act && (nl || nr)) {
                    if (nl) ol = opener.opens(dl, __int_as_float(hl.y), __int_as_float(hl.z));
                    if (nr) orr = opener.opens(dr, __int_as_float(hd.y), __int_as_float(hd.z));
                }
                left = {fc, e.open, __ballot_sync(FULL, ol && act)};
                e = {fc + 1, e.open, __ballot_sync(FULL, orr && act)};
                continue;
            }
        }
        for (; c0 > 0; s0 += kWarp, c0 -= kWarp) {
            const int cn = min(kWarp, c0);
            stage_f32(stage, lane, ft.ph, ft.pl, s0, cn, s1, c1, outside);
            __syncwarp();
            if ((lmask >> lane) & 1u) {
                // per run <= 32 terms, then one Kahan step
                for (int run = 0, first = 0; run < 2; run++) {
                    const int at = run ? s1 : s0, k = run ? c1 : cn, np = rows_for(k);
                    if (k == 0) break;
                    cnt[0] += k - ((unsigned)(me - at) < (unsigned)k);
                    float part[3] = {0.f, 0.f, 0.f};
                    if (soft && unit)
                        rows_f32<DIM, false, true>(stage, first, np, nT, nL, e2h, part);
                    else if (soft)
                        rows_f32<DIM, false, false>(stage, first, np, nT, nL, e2h, part);
                    else
                        rows_f32<DIM, true, false>(stage, first, np, nT, nL, e2h, part);
                    kahan_add_f32<DIM>(part, acc, cmp);
                    first += np;
                }
            }
            __syncwarp();
        }
        if (left.node >= 0) {
            e = left;
            left.node = -1;
        } else if (st.sp == 0) {
            break;
        } else {
            e = st.pop();
        }
        hd = ft.nhdr[e.node];
    }
}

}  // namespace bhut
