// Stable LSD radix sort of (uint64 key, int32 value) pairs.
//
// Replaces np.argsort(codes, kind='stable') of bhut/utils/morton.py:135.  A
// stable order of the keys is unique, so the permutation is bit-identical to
// numpy's.  8-bit digits; keys are cut into tiles of 512 or 2,048 consecutive
// positions (of the order the pass reads).
//
//   k_sort_prep      one read of the keys: every pass's global digit totals
//                    (the totals do not depend on the order) and the first
//                    pass's per-tile digit counts.
//   per pass:
//   k_sort_scan      one block per digit: exclusive scan of that digit's
//                    counts over the tiles, plus the digit's global base
//                    (exclusive prefix of the totals) -> each tile's output
//                    offset for each digit, in stable (tile) order.  Clears
//                    the count table that the scatter below fills.
//   k_sort_scatter   one block per tile: stable rank of every key within the
//                    tile (ballot-based warp multi-split in position order,
//                    warps combined by a per-digit prefix), the tile
//                    reordered by digit in shared memory, then written out in
//                    digit runs, so that consecutive threads store
//                    consecutive addresses.  While writing, it counts the
//                    next pass's digit per destination tile (warp-aggregated
//                    global atomics): the next pass needs no histogram launch.
//
// The fewest keys (sort_sums, common.cuh) go without the scan: each scatter
// block adds up the few tiles' counts itself.  One launch per pass.
//
// No block waits on another block (no look-back): the only cross-block
// dependencies are between launches.  Two launches per pass otherwise.
#include <atomic>
#include <utility>

#include "tree.cuh"

// Points that one block orders (launch_order).  One block / passes, 3-D, us: whole
// rebuilds (captured) of 1,000 points 120 / 133, 2,000 130 / 134, 3,000 147 / 151,
// 4,000 156 / 145; orders 112 / 145, 115 / 149, 128 / 159, 137 / 147; one-shot
// solves of host arrays 211 / 250, 226 / 263, 270 / 296, 302 / 319.  2-D alike: a
// rebuild's graph hides the launches of the passes, so it alone would have the line
// at 3,500.  5,000 points: orders 162 / 161, rebuilds 181 / 156.
#ifndef BHUT_ORDER_SMALL
#define BHUT_ORDER_SMALL 4096
#endif

namespace bhut {

namespace {

constexpr int kWarpsPerTile = kSortThreads / kWarp;    // 8
constexpr int kScanThreads = 256;
static_assert((1 << kSortShiftSmall) % kSortThreads == 0, "tiles of whole blocks");
// resident scatter blocks per SM the register budget must allow (shared
// memory allows five 34 KB tiles of 2,048 keys)
constexpr int kScatterMinBlocks = 4;
static_assert(kScanThreads == kSortThreads, "the scan helper serves both kernels");

template <int TILE>
__device__ __forceinline__ int64_t item_pos(int64_t tile, int warp, int item, int lane)
{
    return tile * TILE + (int64_t)warp * (TILE / kWarpsPerTile) + item * kWarp + lane;
}

// Shared memory of the scatter kernel.
template <int TILE>
struct ScatterSmem {
    uint64_t keys[TILE];
    int32_t vals[TILE];
    uint32_t warp_counts[kWarpsPerTile][256];
    uint32_t delta[256];      // global offset of the digit minus its local offset
    uint32_t local_off[256];
};

// k_sort_prep: block t reads tile t; per-tile counts of digit 0 and the
// global totals of every pass's digit.
template <int SHIFT>
__global__ void __launch_bounds__(kSortThreads)
k_sort_prep(const uint64_t* __restrict__ keys, int64_t n, int passes,
            uint32_t* __restrict__ counts0, int64_t tiles, uint32_t* __restrict__ totals)
{
    constexpr int kTile = 1 << SHIFT, kItems = kTile / kSortThreads;
    __shared__ uint32_t hist[kSortPassesMax][256];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int64_t tile = blockIdx.x;
    for (int p = 0; p < passes; p++) hist[p][tid] = 0;
    __syncthreads();
    // shared-memory atomics; a digit that all lanes of the warp share (ties,
    // or the few distinct high digits of clustered keys) is added once
#pragma unroll 4
    for (int i = 0; i < kItems; i++) {
        const int64_t pos = item_pos<kTile>(tile, warp, i, lane);
        const bool valid = pos < n;
        const unsigned vmask = __ballot_sync(0xffffffffu, valid);
        // (a lane past the end borrows the tile's first key, which exists)
        const uint64_t k = keys[valid ? pos : tile * kTile];
        for (int p = 0; p < passes; p++) {
            const unsigned d = (unsigned)(k >> (8 * p)) & 0xFFu;
            const bool same = __all_sync(0xffffffffu, d == __shfl_sync(0xffffffffu, d, 0));
            if (same) {
                if (lane == 0) atomicAdd(&hist[p][d], (unsigned)__popc(vmask));
            } else if (valid) {
                atomicAdd(&hist[p][d], 1u);
            }
        }
    }
    __syncthreads();
    counts0[(int64_t)tid * tiles + tile] = hist[0][tid];
    for (int p = 0; p < passes; p++) {
        const uint32_t c = hist[p][tid];
        if (c) atomicAdd(&totals[p * 256 + tid], c);
    }
}

// Block-wide exclusive scan of one value per thread (kScanThreads threads).
__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t v, uint32_t* total,
                                                         uint32_t* warp_sums)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp_sums[warp] = x;
    __syncthreads();
    if (warp == 0) {
        uint32_t s = lane < kScanThreads / kWarp ? warp_sums[lane] : 0u;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o) s += y;
        }
        if (lane < kScanThreads / kWarp) warp_sums[lane] = s;
    }
    __syncthreads();
    const uint32_t prefix = (warp > 0 ? warp_sums[warp - 1] : 0u) + x - v;
    if (total) *total = warp_sums[kScanThreads / kWarp - 1];
    __syncthreads();
    return prefix;
}

// k_sort_scan: block d turns row d of the count table (bucket-major: digit d
// of tile t is entry d * tiles + t) into output offsets, and clears row d of
// the next pass's table.
__global__ void __launch_bounds__(kScanThreads)
k_sort_scan(uint32_t* __restrict__ counts, int64_t tiles, const uint32_t* __restrict__ totals,
            uint32_t* __restrict__ next_counts)
{
    __shared__ uint32_t warp_sums[kScanThreads / kWarp];
    __shared__ uint32_t s_base;
    const int d = blockIdx.x, tid = threadIdx.x;
    // base of digit d: sum of the totals of digits below d
    uint32_t below = tid < d ? totals[tid] : 0u;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) below += __shfl_down_sync(0xffffffffu, below, o);
    if (tid == 0) s_base = 0;
    __syncthreads();
    if ((tid & 31) == 0 && below) atomicAdd(&s_base, below);
    __syncthreads();
    uint32_t carry = s_base;
    uint32_t* row = counts + (int64_t)d * tiles;
    uint32_t* nrow = next_counts ? next_counts + (int64_t)d * tiles : nullptr;
    for (int64_t base = 0; base < tiles; base += kScanThreads) {
        const int64_t t = base + tid;
        const uint32_t v = t < tiles ? row[t] : 0u;
        uint32_t total;
        const uint32_t ex = block_exclusive_scan(v, &total, warp_sums);
        if (t < tiles) {
            row[t] = carry + ex;
            if (nrow) nrow[t] = 0u;
        }
        carry += total;
    }
}

// k_sort_scatter: see the file comment.  `next_counts` (may be null) gets
// the digit at `next_shift` of every key, per destination tile.
//
// SUMS (few tiles): no scan launch; `offsets` are the counts themselves, tile
// by tile (entry tile * 256 + digit), which every block adds up, and the block
// clears its part of `clear` (may be null), the table of the pass after next.
template <int SHIFT, bool SUMS>
__global__ void __launch_bounds__(kSortThreads, kScatterMinBlocks)
k_sort_scatter(const uint64_t* __restrict__ keys_in, const int32_t* __restrict__ vals_in,
               uint64_t* __restrict__ keys_out, int32_t* __restrict__ vals_out, int64_t n,
               int shift, const uint32_t* __restrict__ offsets, int64_t tiles,
               uint32_t* __restrict__ next_counts, int next_shift, uint32_t* __restrict__ clear)
{
    constexpr int kTile = 1 << SHIFT, kItems = kTile / kSortThreads;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    ScatterSmem<kTile>& sm = *reinterpret_cast<ScatterSmem<kTile>*>(smem_raw);
    __shared__ uint32_t warp_sums[kSortThreads / kWarp];
    const unsigned FULL = 0xffffffffu;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int64_t tile = blockIdx.x;
#pragma unroll
    for (int w = 0; w < kWarpsPerTile; w++) sm.warp_counts[w][tid] = 0;
    uint32_t before_tile = 0, of_digit = 0;   // keys of digit `tid`
    if (SUMS) {
#pragma unroll 8
        for (int t = 0; t < (int)tiles; t++) {
            const uint32_t c = offsets[t * 256 + tid];
            of_digit += c;
            before_tile += t < tile ? c : 0u;
        }
        if (clear) clear[tile * 256 + tid] = 0u;
    }
    __syncthreads();

    uint64_t k[kItems];
    uint32_t rank[kItems];
    const unsigned lt_mask = (1u << lane) - 1u;
#pragma unroll
    for (int i = 0; i < kItems; i++) {
        const int64_t p = item_pos<kTile>(tile, warp, i, lane);
        const bool valid = p < n;
        k[i] = valid ? keys_in[p] : ~0ull;
        const unsigned d = (unsigned)(k[i] >> shift) & 0xFFu;
        // lanes holding the same digit (warp multi-split by eight ballots)
        unsigned peers = __ballot_sync(FULL, valid);
#pragma unroll
        for (int b = 0; b < 8; b++) {
            const bool bit = (d >> b) & 1u;
            const unsigned bal = __ballot_sync(FULL, bit);
            peers &= bit ? bal : ~bal;
        }
        const uint32_t before = sm.warp_counts[warp][d];
        rank[i] = before + __popc(peers & lt_mask);
        __syncwarp();
        if (valid && (peers & lt_mask) == 0) sm.warp_counts[warp][d] = before + __popc(peers);
        __syncwarp();
    }
    __syncthreads();
    // per digit (thread tid = digit): prefix over warps, then the tile-local
    // digit offsets (exclusive scan over digits)
    uint32_t run = 0;
#pragma unroll
    for (int w = 0; w < kWarpsPerTile; w++) {
        const uint32_t t = sm.warp_counts[w][tid];
        sm.warp_counts[w][tid] = run;
        run += t;
    }
    const uint32_t loc = block_exclusive_scan(run, nullptr, warp_sums);
    sm.local_off[tid] = loc;
    const uint32_t to = SUMS ? block_exclusive_scan(of_digit, nullptr, warp_sums) + before_tile
                             : offsets[(int64_t)tid * tiles + tile];
    sm.delta[tid] = to - loc;
    __syncthreads();
    // reorder the tile by digit in shared memory (stable)
#pragma unroll
    for (int i = 0; i < kItems; i++) {
        const int64_t p = item_pos<kTile>(tile, warp, i, lane);
        if (p < n) {
            const unsigned d = (unsigned)(k[i] >> shift) & 0xFFu;
            const uint32_t lpos = sm.local_off[d] + sm.warp_counts[warp][d] + rank[i];
            if (lpos < (uint32_t)kTile) {   // always true; guards shared memory
                sm.keys[lpos] = k[i];
                sm.vals[lpos] = vals_in[p];    // (read here: fewer live registers)
            }
        }
    }
    __syncthreads();
    // write out in digit runs: position j of the reordered tile goes to
    // delta[digit] + j
    const int64_t cnt = min((int64_t)kTile, n - tile * kTile);
#pragma unroll 4
    for (int j = tid; j < cnt; j += kSortThreads) {
        const uint64_t key = sm.keys[j];
        const unsigned d = (unsigned)(key >> shift) & 0xFFu;
        const uint32_t dst = sm.delta[d] + (uint32_t)j;
        if (dst >= (uint32_t)n) continue;   // always false; guards the output
        keys_out[dst] = key;
        vals_out[dst] = sm.vals[j];
        if (next_counts) {   // warp-aggregated: one atomic per (digit, tile) in the warp
            const unsigned nd = (unsigned)(key >> next_shift) & 0xFFu;
            const unsigned dtile = dst >> SHIFT;
            const unsigned peers = __match_any_sync(__activemask(), (dtile << 8) | nd);
            if ((peers & ((1u << lane) - 1u)) == 0)
                atomicAdd(&next_counts[SUMS ? (int64_t)dtile * 256 + nd : (int64_t)nd * tiles + dtile],
                          (unsigned)__popc(peers));
        }
    }
}

// k_sort_count: digit 0 of every key per tile, for the first pass with SUMS;
// clears the second pass's table.
template <int SHIFT>
__global__ void __launch_bounds__(kSortThreads)
k_sort_count(const uint64_t* __restrict__ keys, int n, uint32_t* __restrict__ counts,
             uint32_t* __restrict__ clear)
{
    __shared__ uint32_t hist[256];
    const int tid = threadIdx.x, tile = blockIdx.x;
    hist[tid] = 0;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < (1 << SHIFT) / kSortThreads; i++) {
        const int p = (tile << SHIFT) + i * kSortThreads + tid;
        if (p < n) atomicAdd(&hist[(unsigned)keys[p] & 0xffu], 1u);
    }
    __syncthreads();
    counts[tile * 256 + tid] = hist[tid];
    clear[tile * 256 + tid] = 0u;
}

struct SortLayout {
    uint64_t* keys_alt;
    int32_t* vals_alt;
    uint32_t* counts[3];
    uint32_t* totals;
};

SortLayout carve(void* scratch, int64_t n)
{
    char* s = (char*)scratch;
    SortLayout L;
    L.keys_alt = (uint64_t*)s; s += sort_align(sizeof(uint64_t) * (size_t)n);
    L.vals_alt = (int32_t*)s;  s += sort_align(sizeof(int32_t) * (size_t)n);
    const size_t table = sizeof(uint32_t) * 256 * (size_t)sort_tiles(n);
    for (int k = 0; k < sort_tables(n); k++) {
        L.counts[k] = (uint32_t*)s;
        s += sort_align(table);
    }
    L.totals = (uint32_t*)s;
    return L;
}

}  // namespace

// ---------------------------------------------------------------------------
// Small inputs: Morton keys, stable sort and Morton-ordered copies by one block.
//
// Up to a few thousand points the passes above take as long as their launches
// (one a pass, 11 with the keys and the gather).  One block holds the keys in
// registers and ranks, scatters and reads them back through shared memory,
// eight bits at a time as above; places past the last point carry the largest
// key and stay behind all others.
// ---------------------------------------------------------------------------
namespace {

constexpr int kSmallThreads = 1024;
constexpr int kSmallWarps = kSmallThreads / kWarp;

template <int ITEMS>
struct SmallSmem {
    uint64_t keys[kSmallThreads * ITEMS];
    uint16_t idx[kSmallThreads * ITEMS];
    uint32_t counts[kSmallWarps][256];
    uint32_t offset[256];
    uint32_t sums[8];
};

template <int DIM, int ITEMS>
__global__ void __launch_bounds__(kSmallThreads)
k_order_small(const double* __restrict__ pos, const double* __restrict__ mass, int n,
              const double* __restrict__ box, uint64_t* __restrict__ keys,
              int32_t* __restrict__ perm, double* __restrict__ sx, double* __restrict__ sy,
              double* __restrict__ sz, double* __restrict__ sm)
{
    static_assert(kSmallThreads * ITEMS <= 65536, "16-bit indices");
    extern __shared__ __align__(16) unsigned char small_raw[];
    SmallSmem<ITEMS>& S = *reinterpret_cast<SmallSmem<ITEMS>*>(small_raw);
    const unsigned FULL = 0xffffffffu;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned below = (1u << lane) - 1u;
    const MortonBox<DIM> mb(box);
    uint64_t k[ITEMS];
    uint32_t id[ITEMS], rank[ITEMS];
#pragma unroll
    for (int i = 0; i < ITEMS; i++) {
        const int p = (warp * ITEMS + i) * kWarp + lane;
        k[i] = p < n ? mb.key(pos, p) : ~0ull;
        id[i] = (uint32_t)p;
    }
    constexpr int kPasses = DIM == 3 ? 8 : 6;   // 63 and 42 key bits
    for (int pass = 0; pass < kPasses; pass++) {
        const int shift = 8 * pass;
        for (int j = tid; j < kSmallWarps * 256; j += kSmallThreads) (&S.counts[0][0])[j] = 0;
        __syncthreads();
#pragma unroll
        for (int i = 0; i < ITEMS; i++) {
            const unsigned d = (unsigned)(k[i] >> shift) & 0xffu;
            unsigned peers = FULL;
#pragma unroll
            for (int b = 0; b < 8; b++) {
                const bool bit = (d >> b) & 1u;
                const unsigned bal = __ballot_sync(FULL, bit);
                peers &= bit ? bal : ~bal;
            }
            const uint32_t before = S.counts[warp][d];
            rank[i] = before + __popc(peers & below);
            __syncwarp();
            if ((peers & below) == 0) S.counts[warp][d] = before + __popc(peers);
            __syncwarp();
        }
        __syncthreads();
        // four threads per digit: prefix over the warps, eight warps each
        const int digit = tid >> 2, part = tid & 3;
        uint32_t c[8], run = 0;
#pragma unroll
        for (int j = 0; j < 8; j++) {
            c[j] = run;
            run += S.counts[8 * part + j][digit];
        }
        uint32_t x = run;
#pragma unroll
        for (int o = 1; o < 4; o <<= 1) {
            const uint32_t y = __shfl_up_sync(FULL, x, o);
            if (part >= o) x += y;
        }
        const uint32_t first = x - run;
#pragma unroll
        for (int j = 0; j < 8; j++) S.counts[8 * part + j][digit] = first + c[j];
        if (part == 3) S.offset[digit] = x;
        __syncthreads();
        uint32_t v = 0, inc = 0;
        if (tid < 256) {   // exclusive scan over the digits
            v = inc = S.offset[tid];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(FULL, inc, o);
                if (lane >= o) inc += y;
            }
            if (lane == 31) S.sums[warp] = inc;
        }
        __syncthreads();
        if (tid < 256) {
            uint32_t base = 0;
            for (int w = 0; w < warp; w++) base += S.sums[w];
            S.offset[tid] = base + inc - v;
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < ITEMS; i++) {
            const unsigned d = (unsigned)(k[i] >> shift) & 0xffu;
            const uint32_t at = S.offset[d] + S.counts[warp][d] + rank[i];
            S.keys[at] = k[i];
            S.idx[at] = (uint16_t)id[i];
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < ITEMS; i++) {
            const int p = (warp * ITEMS + i) * kWarp + lane;
            k[i] = S.keys[p];
            id[i] = S.idx[p];
        }
        // (the next pass writes keys only after its barriers)
    }
#pragma unroll
    for (int i = 0; i < ITEMS; i++) {
        const int p = (warp * ITEMS + i) * kWarp + lane;
        if (p >= n) continue;
        const int64_t q = id[i];
        keys[p] = k[i];
        perm[p] = (int32_t)q;
        if (sx) {
            sx[p] = pos[q * DIM];
            sy[p] = pos[q * DIM + 1];
            sz[p] = DIM == 3 ? pos[q * DIM + 2] : 0.0;
            if (mass) sm[p] = mass[q];
        }
    }
}

template <int DIM, int ITEMS>
int run_order_small(const double* pos, const double* mass, int n, const double* box,
                    uint64_t* keys, int32_t* perm, double* sx, double* sy, double* sz, double* sm,
                    cudaStream_t stream)
{
    static std::atomic<bool> smem_set[64];
    int dev = 0;
    BHUT_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64 || !smem_set[dev].load(std::memory_order_acquire)) {
        BHUT_CUDA(cudaFuncSetAttribute(k_order_small<DIM, ITEMS>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)sizeof(SmallSmem<ITEMS>)));
        if (dev >= 0 && dev < 64) smem_set[dev].store(true, std::memory_order_release);
    }
    k_order_small<DIM, ITEMS><<<1, kSmallThreads, sizeof(SmallSmem<ITEMS>), stream>>>(
        pos, mass, n, box, keys, perm, sx, sy, sz, sm);
    BHUT_CUDA(cudaGetLastError());
    note_launches(1);
    return kOk;
}

template <int DIM>
int order_small(const double* pos, const double* mass, int n, const double* box, uint64_t* keys,
                int32_t* perm, double* sx, double* sy, double* sz, double* sm, cudaStream_t s)
{
    if (n <= 1024) return run_order_small<DIM, 1>(pos, mass, n, box, keys, perm, sx, sy, sz, sm, s);
    if (n <= 2048) return run_order_small<DIM, 2>(pos, mass, n, box, keys, perm, sx, sy, sz, sm, s);
    return run_order_small<DIM, 4>(pos, mass, n, box, keys, perm, sx, sy, sz, sm, s);
}

}  // namespace

int launch_order(const double* pos, const double* mass, int64_t n, int dim, const double* box,
                 uint64_t* keys, int32_t* perm, double* sx, double* sy, double* sz, double* sm,
                 void* scratch, cudaStream_t s)
{
    static_assert(BHUT_ORDER_SMALL <= kSmallThreads * 4, "the largest block");
    if (n <= BHUT_ORDER_SMALL)
        return dim == 3 ? order_small<3>(pos, mass, (int)n, box, keys, perm, sx, sy, sz, sm, s)
                        : order_small<2>(pos, mass, (int)n, box, keys, perm, sx, sy, sz, sm, s);
    BHUT_TRY(launch_morton(pos, n, dim, box, keys, perm, s));
    BHUT_TRY(radix_sort_pairs(keys, perm, n, dim == 3 ? 63 : 42, scratch, s));
    return sx ? launch_gather(pos, mass, perm, n, dim, sx, sy, sz, sm, s) : kOk;
}

namespace {

// An odd number of passes ends in the other buffers.
int copy_back(uint64_t* keys, int32_t* vals, const uint64_t* kin, const int32_t* vin, int64_t n,
              cudaStream_t stream)
{
    if (kin == keys) return kOk;
    BHUT_CUDA(cudaMemcpyAsync(keys, kin, sizeof(uint64_t) * (size_t)n, cudaMemcpyDeviceToDevice, stream));
    BHUT_CUDA(cudaMemcpyAsync(vals, vin, sizeof(int32_t) * (size_t)n, cudaMemcpyDeviceToDevice, stream));
    return kOk;
}

struct SortArgs {
    uint64_t* keys;
    int32_t* vals;
    int64_t n, tiles;
    int passes;
    SortLayout L;
    cudaStream_t stream;
};

// One launch a pass (sort_sums).
int sort_with_sums(const SortArgs& a)
{
    constexpr int S = kSortShiftSmall, smem = (int)sizeof(ScatterSmem<1 << S>);
    static_assert(smem <= 48 * 1024, "within the default limit");
    const unsigned tiles = (unsigned)a.tiles;
    const SortLayout& L = a.L;
    k_sort_count<S><<<tiles, kSortThreads, 0, a.stream>>>(a.keys, (int)a.n, L.counts[0], L.counts[1]);
    uint64_t *kin = a.keys, *kout = L.keys_alt;
    int32_t *vin = a.vals, *vout = L.vals_alt;
    for (int pass = 0; pass < a.passes; pass++) {
        k_sort_scatter<S, true><<<tiles, kSortThreads, smem, a.stream>>>(
            kin, vin, kout, vout, a.n, 8 * pass, L.counts[pass % 3], a.tiles,
            pass + 1 < a.passes ? L.counts[(pass + 1) % 3] : nullptr, 8 * (pass + 1),
            pass + 2 < a.passes ? L.counts[(pass + 2) % 3] : nullptr);
        std::swap(kin, kout);
        std::swap(vin, vout);
    }
    BHUT_CUDA(cudaGetLastError());
    note_launches(1 + (int64_t)a.passes);
    return copy_back(a.keys, a.vals, kin, vin, a.n, a.stream);
}

// A scan and a scatter a pass.
template <int SHIFT>
int sort_with_scans(const SortArgs& a)
{
    // the scatter's shared memory may exceed the default limit, and wants all
    // of the unified L1/shared storage (several tiles per SM): once per device
    const auto scatter = k_sort_scatter<SHIFT, false>;
    constexpr int smem = (int)sizeof(ScatterSmem<1 << SHIFT>);
    {
        static std::atomic<bool> smem_set[64];
        int dev = 0;
        BHUT_CUDA(cudaGetDevice(&dev));
        if (dev < 0 || dev >= 64 || !smem_set[dev].load(std::memory_order_acquire)) {
            BHUT_CUDA(cudaFuncSetAttribute(scatter, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           smem));
            BHUT_CUDA(cudaFuncSetAttribute(scatter, cudaFuncAttributePreferredSharedMemoryCarveout,
                                           (int)cudaSharedmemCarveoutMaxShared));
            if (dev >= 0 && dev < 64) smem_set[dev].store(true, std::memory_order_release);
        }
    }
    const unsigned tiles = (unsigned)a.tiles;
    const SortLayout& L = a.L;
    BHUT_CUDA(cudaMemsetAsync(L.totals, 0, sizeof(uint32_t) * 256 * kSortPassesMax, a.stream));
    k_sort_prep<SHIFT><<<tiles, kSortThreads, 0, a.stream>>>(a.keys, a.n, a.passes, L.counts[0],
                                                             a.tiles, L.totals);
    uint64_t *kin = a.keys, *kout = L.keys_alt;
    int32_t *vin = a.vals, *vout = L.vals_alt;
    for (int pass = 0; pass < a.passes; pass++) {
        const bool last = pass + 1 == a.passes;
        uint32_t* cur = L.counts[pass & 1];
        uint32_t* nxt = last ? nullptr : L.counts[(pass + 1) & 1];
        k_sort_scan<<<256, kScanThreads, 0, a.stream>>>(cur, a.tiles, L.totals + 256 * pass, nxt);
        scatter<<<tiles, kSortThreads, smem, a.stream>>>(
            kin, vin, kout, vout, a.n, 8 * pass, cur, a.tiles, nxt, 8 * (pass + 1), nullptr);
        std::swap(kin, kout);
        std::swap(vin, vout);
    }
    BHUT_CUDA(cudaGetLastError());
    note_launches(1 + 2ll * a.passes);
    return copy_back(a.keys, a.vals, kin, vin, a.n, a.stream);
}

}  // namespace

int radix_sort_pairs(uint64_t* keys, int32_t* vals, int64_t n, int bits, void* scratch,
                     cudaStream_t stream)
{
    if (n <= 1) return kOk;
    if (n > 0x7fffffffLL) { set_error("radix sort supports at most 2^31-1 keys"); return kInvalid; }
    const int passes = (bits + 7) / 8;
    if (passes < 1 || passes > kSortPassesMax) {
        set_error("radix sort: %d key bits out of range", bits);
        return kInvalid;
    }
    const SortArgs a{keys, vals, n, sort_tiles(n), passes, carve(scratch, n), stream};
    static_assert(BHUT_SORT_SUMS_MAX <= BHUT_SORT_SMALL_TILE_MAX, "sums add up small tiles");
    if (sort_sums(n)) return sort_with_sums(a);
    return sort_small_tiles(n) ? sort_with_scans<kSortShiftSmall>(a) : sort_with_scans<kSortShift>(a);
}

}  // namespace bhut
