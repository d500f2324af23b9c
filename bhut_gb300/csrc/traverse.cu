// Barnes-Hut traversal, FP64 "exact" form, and the FP64 direct-sum kernel.
//
// k_traverse_exact replaces the per-target loop of bhut/traverse/bh.py:
// _barnes_hut_single_target (:485-548, self) and
// _barnes_hut_single_target_external (:83-146).  One warp owns 32
// Morton-contiguous targets and walks the tree with a shared stack of
// (node, lane mask) entries: a lane that accepts a node adds its monopole and
// drops out of that subtree, so every lane visits exactly the nodes of the
// reference's own traversal for its target, right child first (bh.py:531-537).
// Contributions are summed in that order within the subtrees at the depth
// top_levels (a function of the node count alone), and these sums in pairs,
// child by child, up to the root: whichever levels the warps of a call split,
// a target's value depends on the tree only.  Per-pair arithmetic is the Numba leaf
// loop (bh.py:226-280) with explicit round-to-nearest intrinsics and IEEE
// sqrt/division, so P2P terms match the reference's bit for bit; monopoles
// use r2^1.5 = r2 * sqrt(r2) in place of pow (kernels.py:66), within 2 ulp.
// Products, square roots and reciprocals run on the integer and FP32 pipes
// (fp64int.cuh), correctly rounded all the same; the FP64 pipe keeps a pair's
// nine additions.  100k Plummer traversal 243 -> 96 ms, direct sum of 20,000
// 28.6 -> 9.4 ms, bit for bit the same (with the products left to the FP64 pipe
// 138 and 16.2 ms).  Bound now by the ALU and FP64 pipes, 71 and 70 % busy.
#include "fp64int.cuh"
#include "tree.cuh"

namespace bhut {

constexpr int kTravWarps = 4;
constexpr int kTravThreads = kTravWarps * kWarp;

// Resident blocks per SM of k_traverse_exact, at the registers that they allow.
// 3-D, split: without a bound (101 registers, 4 blocks) / 5 / 6: 100k Plummer
// 93.2 / 85.7 / 82.5 ms, 10k 1.97 / 1.83 / 1.76; not split, 5 / 6: 200k 140 / 145.
// 2-D, 6 / 7: 50k 3.68 / 3.60, 10k 0.80 / 0.78, targets of either 0 to 6 % less / more.
constexpr int exact_blocks(int dim, bool split) { return dim == 3 && !split ? 5 : 6; }

// v, kept in registers (a product of two kernel arguments would otherwise be
// formed again for every pair).
static __device__ __forceinline__ double held(double v)
{
    asm volatile("" : "+d"(v));
    return v;
}

// The leaf loop's force (bh.py:262-278) in FP64 instructions; false: none
// (r^2 + eps^2 == 0).
template <int DIM>
static __device__ __noinline__ bool pair_fp64_force(double dx, double dy, double dz, double gm,
                                                    double eps2, double3* F)
{
    double r2 = __dmul_rn(dx, dx);
    r2 = __dadd_rn(r2, __dmul_rn(dy, dy));
    if (DIM == 3) r2 = __dadd_rn(r2, __dmul_rn(dz, dz));
    r2 = __dadd_rn(r2, eps2);
    if (r2 == 0.0) return false;
    const double ri = __ddiv_rn(1.0, __dsqrt_rn(r2));
    const double f = __dmul_rn(gm, __dmul_rn(__dmul_rn(ri, ri), ri));
    F->x = __dmul_rn(f, dx);
    F->y = __dmul_rn(f, dy);
    F->z = DIM == 3 ? __dmul_rn(f, dz) : 0.0;
    return true;
}

// The leaf loop's term at displacement (dx, dy, dz), added to (ax, ay, az);
// gm = G m.  Returns whether it counts (r^2 + eps^2 != 0).
template <int DIM>
static __device__ __forceinline__ bool pair_exact(double dx, double dy, double dz, double gm,
                                                  double eps2, double& ax, double& ay, double& az)
{
    using fp64int::parts;
    using fp64int::within;
    // ranges in which no product below leaves the normal numbers: |d| within
    // 2^+-250, |G m| within 2^+-200, r^2 + eps^2 within 2^-340 .. 2^300
    const auto X = parts(dx), Y = parts(dy), Z = parts(DIM == 3 ? dz : 0.0), M = parts(gm);
    bool ok = within(X, -250, 250) && within(Y, -250, 250) && within(Z, -250, 250) &&
              within(M, -200, 200);
    // (100k Plummer traversal with all products in integers 95.9 ms, the squares
    // alone 103.3, the forces alone 104.9, neither 122.4)
    double r2 = fp64int::mul(X, X);
    r2 = __dadd_rn(r2, fp64int::mul(Y, Y));
    if (DIM == 3) r2 = __dadd_rn(r2, fp64int::mul(Z, Z));
    r2 = __dadd_rn(r2, eps2);
    const auto R = parts(r2);
    if (ok && R.zero) return false;   // (never -0)
    ok = ok && within(R, -340, 300);
    const auto I = fp64int::rsqrt(R);
    const auto W = fp64int::product(M, fp64int::product(fp64int::product(I, I), I));
    double3 F = make_double3(fp64int::mul(W, X), fp64int::mul(W, Y),
                             DIM == 3 ? fp64int::mul(W, Z) : 0.0);
    if (!ok) {   // something beyond those ranges
        double3 G;
        if (!pair_fp64_force<DIM>(dx, dy, dz, gm, eps2, &G)) return false;
        F = G;
    }
    ax = __dadd_rn(ax, F.x);
    ay = __dadd_rn(ay, F.y);
    if (DIM == 3) az = __dadd_rn(az, F.z);
    return true;
}

// size / sqrt(s) >= theta (bh.py:576-601) for s = |x - com|^2 as np.linalg.norm
// sums it (fma chain, OpenBLAS ddot).  The squares decide outside 2^-39 of
// each other (both sides are within a few 2^-53 of the exact ones, and
// positive doubles order as integers); inside, or outside the normal range, or
// for a negative theta or size (tree statistics and imported trees take both),
// the reference's own square root and division.
static __device__ __forceinline__ bool opens(double s, double size, double theta)
{
    const int64_t a = (int64_t)fp64int::bits(__dmul_rn(size, size));
    const int64_t b = (int64_t)fp64int::bits(__dmul_rn(__dmul_rn(theta, theta), s));
    const int64_t gap = a - b;
    const bool negative = (int64_t)(fp64int::bits(size) | fp64int::bits(theta)) < 0;
    if ((gap > 8192 || gap < -8192) && !negative && fp64int::normal_positive(a) &&
        fp64int::normal_positive(b))
        return gap > 0;
    const double d = __dsqrt_rn(s);
    return d == 0.0 || __ddiv_rn(size, d) >= theta;
}

template <int DIM>
static __device__ __forceinline__ double norm2_fma(double dx, double dy, double dz)
{
    const double s = __fma_rn(dy, dy, __dmul_rn(dx, dx));
    return DIM == 3 ? __fma_rn(dz, dz, s) : s;
}

template <int DIM>
__device__ __forceinline__ bool open_exact(double x, double y, double z, NodeCM cm, double size,
                                           double theta)
{
    return opens(norm2_fma<DIM>(__dsub_rn(x, cm.x), __dsub_rn(y, cm.y),
                                DIM == 3 ? __dsub_rn(z, cm.z) : 0.0), size, theta);
}

// kernels.py:52-69 acc_monopole (single vector) via acc_monopole_node, at
// displacement (dx, dy, dz) from the target.
template <int DIM>
__device__ __forceinline__ void monopole_exact(double dx, double dy, double dz, double m,
                                               double eps2, double G, double& ax, double& ay,
                                               double& az)
{
    double r2 = __dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy));
    if (DIM == 3) r2 = __dadd_rn(r2, __dmul_rn(dz, dz));
    double r2s = __dadd_rn(r2, eps2);
    if (r2s == 0.0) return;
    double f = __ddiv_rn(__dmul_rn(G, m), __dmul_rn(r2s, fp64int::sqrt(r2s)));
    ax = __dadd_rn(ax, __dmul_rn(f, dx));
    ay = __dadd_rn(ay, __dmul_rn(f, dy));
    if (DIM == 3) az = __dadd_rn(az, __dmul_rn(f, dz));
}

// SPLIT: 2^levels warps share 32 targets as in k_traverse_fast (few targets;
// a warp follows the bits of its path through the top levels and walks the
// subtree it reaches); levels <= top.
//
// The walk keeps the place (d, idx) of the unit that it is summing: a node above
// depth `top`, or a subtree at that depth.  At a unit's end the sum waits in
// saved[d] when it is a right child's, for its left sibling's; a left child's is
// added to it and the pair is the parent's.  Lanes without a part in a unit add
// zeros.
template <int DIM, bool SPLIT>
__global__ void __launch_bounds__(kTravThreads, exact_blocks(DIM, SPLIT))
k_traverse_exact(TreeDev t, const double* __restrict__ tx, const double* __restrict__ ty,
                 const double* __restrict__ tz, const int32_t* __restrict__ self_id,
                 const int32_t* __restrict__ out_idx, int64_t nt, double theta, double eps,
                 double G, double* __restrict__ out, unsigned* __restrict__ err,
                 unsigned long long* __restrict__ stats, int levels0, int top,
                 double* __restrict__ partial)
{
    __shared__ int2 stack[kTravWarps][kStackDepth];
    __shared__ double px[kTravWarps][kWarp], py[kTravWarps][kWarp], pz[kTravWarps][kWarp],
        pm[kTravWarps][kWarp];
    __shared__ int32_t pid[kTravWarps][kWarp];
    __shared__ double sum[SPLIT ? kTravWarps : 1][SPLIT ? DIM : 1][kWarp];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const double eps2 = held(__dmul_rn(eps, eps));
    const unsigned FULL = 0xffffffffu;

    const int shares = SPLIT ? (1 << levels0) / kTravWarps : 1;   // blocks per group
    const int64_t step = SPLIT ? gridDim.x / shares : (int64_t)gridDim.x * kTravWarps;
    const int share = SPLIT ? (int)(blockIdx.x % (unsigned)shares) : 0;

    for (int64_t g = SPLIT ? blockIdx.x / (unsigned)shares
                           : (int64_t)blockIdx.x * kTravWarps + w;
         g * kWarp < nt; g += step) {
        const int64_t i = g * kWarp + lane;
        const int path = SPLIT ? share * kTravWarps + w : 0;
        bool own = path == 0;                                // works on the node
        const bool valid = i < nt;
        const double x = valid ? tx[i] : 0.0, y = valid ? ty[i] : 0.0;
        const double z = (valid && DIM == 3) ? tz[i] : 0.0;
        const int32_t me = (valid && self_id) ? self_id[i] : -1;
        double ax = 0.0, ay = 0.0, az = 0.0;
        double saved[kTopLevels + 1][DIM];
        int d = 0, idx = 0, sp0 = 0;
        bool fresh = true;                                   // the next node begins a unit
        unsigned long long n_p2p = 0, n_m2p = 0, n_visit = 0;
        const unsigned live = __ballot_sync(FULL, valid);
        if (lane == 0) stack[w][0] = make_int2(0, (int)live);
        int sp = 1;
        bool overflow = false;
        __syncwarp();
        while (sp > 0) {
            const int2 e = stack[w][--sp];
            __syncwarp();
            if (fresh) sp0 = sp;
            unsigned omask = 0;
            const int node = e.x;
            const unsigned mask = (unsigned)e.y;
            const bool act = (mask >> lane) & 1u;
            n_visit += act && own;
            const NodeCM cm = t.cm[node];
            const int fc = t.first_child[node];
            if (cm.w == 0.0) {                               // bh.py:514
            } else if (fc < 0) {                             // leaf: bh.py:520-524
                const int s = t.start[node], c = own ? t.count[node] : 0;
                double lx = 0.0, ly = 0.0, lz = 0.0;
                for (int b = 0; b < c; b += kWarp) {
                    const int jj = b + lane;
                    if (jj < c) {
                        px[w][lane] = t.sx[s + jj];
                        py[w][lane] = t.sy[s + jj];
                        if (DIM == 3) pz[w][lane] = t.sz[s + jj];
                        pm[w][lane] = __dmul_rn(G, t.sm[s + jj]);
                        pid[w][lane] = t.perm[s + jj];
                    }
                    __syncwarp();
                    const int cnt = min(kWarp, c - b);
                    if (act) {
#pragma unroll 1
                        for (int q = 0; q < cnt; q++) {
                            if (pid[w][q] == me) continue;   // self skip, bh.py:254
                            n_p2p += pair_exact<DIM>(
                                __dsub_rn(px[w][q], x), __dsub_rn(py[w][q], y),
                                DIM == 3 ? __dsub_rn(pz[w][q], z) : 0.0, pm[w][q], eps2, lx, ly,
                                lz);
                        }
                    }
                    __syncwarp();
                }
                if (act && own) {
                    ax = __dadd_rn(ax, lx);
                    ay = __dadd_rn(ay, ly);
                    az = __dadd_rn(az, lz);
                }
            } else {                                         // internal: bh.py:525-546
                bool open = false;
                double dx = 0.0, dy = 0.0, dz = 0.0;
                if (act) {
                    dx = __dsub_rn(cm.x, x);
                    dy = __dsub_rn(cm.y, y);
                    if (DIM == 3) dz = __dsub_rn(cm.z, z);
                    open = opens(norm2_fma<DIM>(dx, dy, dz), t.size[node], theta);
                }
                omask = __ballot_sync(FULL, act && open);
                if (act && !open && own) {
                    monopole_exact<DIM>(dx, dy, dz, cm.w, eps2, G, ax, ay, az);
                    n_m2p++;
                }
                if (SPLIT && omask && d < levels0) {
                    const int rest = levels0 - 1 - d;        // bits of the path below the child
                    own = (path & ((1 << rest) - 1)) == 0;
                    if (lane == 0)
                        stack[w][sp] = make_int2(fc + ((path >> rest) & 1), (int)omask);
                    sp++;
                    __syncwarp();
                } else if (omask) {
                    if (sp + 2 > kStackDepth) { overflow = true; break; }
                    if (lane == 0) {
                        stack[w][sp] = make_int2(fc, (int)omask);        // left pushed first
                        stack[w][sp + 1] = make_int2(fc + 1, (int)omask); // right pops first
                    }
                    sp += 2;
                    __syncwarp();
                }
            }
            if (omask && d < top) {                          // on to its (right) child
                idx = 2 * idx + 1;                           // (above levels0 not looked at)
                d++;
                fresh = true;
            } else if ((fresh = sp == sp0)) {                // the unit's end
                double v[3] = {ax, ay, az};
                for (; d > levels0 && !(idx & 1); idx >>= 1, d--) {
#pragma unroll
                    for (int k = 0; k < DIM; k++) v[k] = __dadd_rn(saved[d][k], v[k]);
                }
                const bool wait = d > levels0;
                if (wait) {
#pragma unroll
                    for (int k = 0; k < DIM; k++) saved[d][k] = v[k];
                }
                idx--;
                ax = wait ? 0.0 : v[0];
                ay = wait ? 0.0 : v[1];
                az = wait ? 0.0 : v[2];
            }
        }
        if (overflow && lane == 0) atomicOr(err, kErrStackOverflow);
        if (stats) {
            for (int o = 16; o > 0; o >>= 1) {
                n_p2p += __shfl_down_sync(FULL, n_p2p, o);
                n_m2p += __shfl_down_sync(FULL, n_m2p, o);
                n_visit += __shfl_down_sync(FULL, n_visit, o);
            }
            if (lane == 0) {
                atomicAdd(&stats[0], n_p2p);
                atomicAdd(&stats[1], n_m2p);
                atomicAdd(&stats[2], n_visit);
            }
        }
        if (SPLIT) {
            sum[SPLIT ? w : 0][0][lane] = ax;
            sum[SPLIT ? w : 0][SPLIT ? 1 : 0][lane] = ay;
            if (DIM == 3) sum[SPLIT ? w : 0][SPLIT ? DIM - 1 : 0][lane] = az;
            __syncthreads();
            if (w < DIM && valid) {
                const auto of = [&](int u) { return sum[SPLIT ? u : 0][SPLIT ? w : 0][lane]; };
                const double v = __dadd_rn(__dadd_rn(of(0), of(1)), __dadd_rn(of(2), of(3)));
                if (shares > 1) partial[((int64_t)share * nt + i) * DIM + w] = v;
                else out[(out_idx ? out_idx[i] : i) * DIM + w] = v;
            }
            __syncthreads();
        } else if (valid) {
            const int64_t o = out_idx ? out_idx[i] : i;
            out[o * DIM] = ax;
            out[o * DIM + 1] = ay;
            if (DIM == 3) out[o * DIM + 2] = az;
        }
    }
}

// FP64 direct sum (the theta = 0 limit of the reference; pair arithmetic of
// bh.py:262-278).  Targets given as AoS; self_id[i] >= 0 excludes that
// source.  Sources are staged through shared memory in tiles.  Block
// (x, y) handles targets [256x, 256x + 256) against source chunk y; with
// more than one chunk, per-chunk partial sums go to `partial` and
// k_direct_reduce adds them in chunk order (deterministic).
constexpr int kDirectThreads = 256;
// Sources per chunk, at least: small sums need the blocks (2,000 / 5,000 /
// 20,000 particles, ms: 4096 2.59 / 3.20 / 10.6, 1024 1.47 / 1.48 / 9.4, 512
// 0.91 / 1.23 / 9.4, 256 0.64 / 1.01 / 9.4).
#ifndef BHUT_DIRECT_CHUNK
#define BHUT_DIRECT_CHUNK 256
#endif
constexpr int64_t kDirectChunk = BHUT_DIRECT_CHUNK;

template <int DIM>
__global__ void __launch_bounds__(kDirectThreads)
k_direct(const double* __restrict__ pos, const double* __restrict__ mass, int64_t n,
         const double* __restrict__ targets, const int64_t* __restrict__ self_id, int64_t nt,
         double eps, double G, int64_t chunk, double* __restrict__ out)
{
    __shared__ double sx[kDirectThreads], sy[kDirectThreads], sz[kDirectThreads],
        sm[kDirectThreads];
    const int64_t i = blockIdx.x * (int64_t)kDirectThreads + threadIdx.x;
    const bool valid = i < nt;
    const int64_t me = (valid && self_id) ? self_id[i] : -1;
    double x = 0.0, y = 0.0, z = 0.0;
    if (valid) {
        const double* p = self_id ? pos + me * DIM : targets + i * DIM;
        x = p[0];
        y = p[1];
        if (DIM == 3) z = p[2];
    }
    const double eps2 = held(__dmul_rn(eps, eps));
    double ax = 0.0, ay = 0.0, az = 0.0;
    const int64_t j0 = (int64_t)blockIdx.y * chunk;
    const int64_t j1 = j0 + chunk < n ? j0 + chunk : n;
    for (int64_t b = j0; b < j1; b += kDirectThreads) {
        const int64_t j = b + threadIdx.x;
        __syncthreads();
        if (j < j1) {
            sx[threadIdx.x] = pos[j * DIM];
            sy[threadIdx.x] = pos[j * DIM + 1];
            sz[threadIdx.x] = DIM == 3 ? pos[j * DIM + 2] : 0.0;
            sm[threadIdx.x] = __dmul_rn(G, mass[j]);
        }
        __syncthreads();
        const int cnt = (int)((j1 - b) < kDirectThreads ? (j1 - b) : kDirectThreads);
        if (valid) {
#pragma unroll 1
            for (int q = 0; q < cnt; q++) {
                if (b + q == me) continue;
                pair_exact<DIM>(__dsub_rn(sx[q], x), __dsub_rn(sy[q], y),
                                DIM == 3 ? __dsub_rn(sz[q], z) : 0.0, sm[q], eps2, ax, ay, az);
            }
        }
    }
    if (valid) {
        double* o = out + ((int64_t)blockIdx.y * nt + i) * DIM;
        o[0] = ax;
        o[1] = ay;
        if (DIM == 3) o[2] = az;
    }
}

__global__ void k_direct_reduce(const double* __restrict__ partial, int64_t nt, int dim,
                                int chunks, double* __restrict__ out)
{
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < nt * dim;
         k += (int64_t)gridDim.x * blockDim.x) {
        double s = partial[k];
        for (int c = 1; c < chunks; c++) s = __dadd_rn(s, partial[(int64_t)c * nt * dim + k]);
        out[k] = s;
    }
}

int launch_traverse_exact(const TreeDev& t, const double* tx, const double* ty, const double* tz,
                          const int32_t* self_id, const int32_t* out_idx, int64_t nt, double theta,
                          double eps, double G, double* out, unsigned* err,
                          unsigned long long* stats, cudaStream_t s, int levels, double* partial)
{
    if (nt <= 0) return kOk;
    const int top = top_levels(t.m);
    if (levels > top) { set_error("split deeper than the sums of form exact"); return kInternal; }
    const int64_t groups = (nt + kWarp - 1) / kWarp;
    const int shares = levels > 0 ? (1 << levels) / kTravWarps : 1;
    const unsigned grid = levels > 0 ? (unsigned)(groups * shares)
                                     : grid_for(groups, kTravWarps, 152u * 64u);
    auto* kernel = t.dim == 3
                       ? (levels > 0 ? k_traverse_exact<3, true> : k_traverse_exact<3, false>)
                       : (levels > 0 ? k_traverse_exact<2, true> : k_traverse_exact<2, false>);
    kernel<<<grid, kTravThreads, 0, s>>>(t, tx, ty, tz, self_id, out_idx, nt, theta, eps, G, out,
                                         err, stats, levels, top, partial);
    BHUT_CUDA(cudaGetLastError());
    note_launches(1);
    return shares > 1 ? launch_split_sum(partial, nt, t.dim, shares, true, out_idx, out, s) : kOk;
}

// ---------------------------------------------------------------------------
// Operation counts of compute_tree_statistics (bhut/traverse/bh.py:604-700)
// over any TreeData arrays: per target, nodes popped (empty and out-of-range
// ones included), count - 1 particles for every visited non-empty leaf, and
// accepted internal nodes; opening test of bh.py:576-601 (open_exact).
// One thread per target, private stack; totals summed with warp shuffles and
// one 64-bit atomic per warp and counter.
// ---------------------------------------------------------------------------
constexpr int kStatStack = 128;

template <int DIM>
__global__ void __launch_bounds__(256)
k_tree_statistics(StatTree t, const double* __restrict__ tg, int64_t nt, double theta,
                  unsigned long long* __restrict__ totals, unsigned* __restrict__ err)
{
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    unsigned long long nodes = 0, parts = 0, monos = 0;
    if (i < nt) {
        const double x = tg[i * DIM], y = tg[i * DIM + 1], z = DIM == 3 ? tg[i * DIM + 2] : 0.0;
        int64_t stack[kStatStack];
        int sp = 0;
        stack[sp++] = 0;
        while (sp > 0) {
            const int64_t k = stack[--sp];
            nodes++;
            if (k < 0 || k >= t.m || t.mass[k] == 0.0) continue;
            const int64_t fc = t.first_child[k];
            if (fc == -1) {
                const int64_t c = t.count[k];
                if (t.start[k] != -1 && c > 0) parts += (unsigned long long)(c - 1);
                continue;
            }
            NodeCM cm;
            cm.x = t.com[k * DIM];
            cm.y = t.com[k * DIM + 1];
            cm.z = DIM == 3 ? t.com[k * DIM + 2] : 0.0;
            cm.w = 0.0;
            if (open_exact<DIM>(x, y, z, cm, __dmul_rn(2.0, t.half_size[k]), theta)) {
                const int64_t nc = t.child_count[k];
                if (sp + nc > kStatStack) {
                    atomicOr(err, kErrStackOverflow);
                    break;
                }
                for (int64_t j = 0; j < nc; j++) stack[sp++] = fc + j;
            } else {
                monos++;
            }
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        nodes += __shfl_down_sync(0xffffffffu, nodes, o);
        parts += __shfl_down_sync(0xffffffffu, parts, o);
        monos += __shfl_down_sync(0xffffffffu, monos, o);
    }
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(&totals[0], nodes);
        atomicAdd(&totals[1], parts);
        atomicAdd(&totals[2], monos);
    }
}

int launch_tree_statistics(const StatTree& t, int dim, const double* targets, int64_t nt,
                           double theta, unsigned long long* totals, unsigned* err,
                           cudaStream_t s)
{
    BHUT_CUDA(cudaMemsetAsync(totals, 0, sizeof(unsigned long long) * 3, s));
    if (nt <= 0) return kOk;
    const unsigned grid = (unsigned)((nt + 255) / 256);
    if (dim == 3) k_tree_statistics<3><<<grid, 256, 0, s>>>(t, targets, nt, theta, totals, err);
    else k_tree_statistics<2><<<grid, 256, 0, s>>>(t, targets, nt, theta, totals, err);
    BHUT_CUDA(cudaGetLastError());
    note_launches(1);
    return kOk;
}

int direct_chunks(int64_t n, int64_t nt)
{
    const int64_t tblocks = (nt + kDirectThreads - 1) / kDirectThreads;
    int64_t want = (152 * 8 + tblocks - 1) / tblocks;        // fill the GPU ~8 blocks per SM
    int64_t maxc = (n + kDirectChunk - 1) / kDirectChunk;
    int64_t c = want < maxc ? want : maxc;
    return (int)(c < 1 ? 1 : (c > 1024 ? 1024 : c));
}

int launch_direct(const double* pos, const double* mass, int64_t n, int dim, const double* targets,
                  const int64_t* self_id, int64_t nt, double eps, double G, double* out,
                  double* partial, int chunks, cudaStream_t s)
{
    if (nt <= 0) return kOk;
    const int64_t chunk = (n + chunks - 1) / chunks;
    dim3 grid((unsigned)((nt + kDirectThreads - 1) / kDirectThreads), (unsigned)chunks);
    double* dst = chunks > 1 ? partial : out;
    if (dim == 3)
        k_direct<3><<<grid, kDirectThreads, 0, s>>>(pos, mass, n, targets, self_id, nt, eps, G, chunk,
                                                    dst);
    else
        k_direct<2><<<grid, kDirectThreads, 0, s>>>(pos, mass, n, targets, self_id, nt, eps, G, chunk,
                                                    dst);
    if (chunks > 1)
        k_direct_reduce<<<grid_for(nt * dim, 256), 256, 0, s>>>(partial, nt, dim, chunks, out);
    BHUT_CUDA(cudaGetLastError());
    note_launches(chunks > 1 ? 2 : 1);
    return kOk;
}

}  // namespace bhut
