// Shared definitions for the GB300 Barnes-Hut engine (sm_103a).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace bhut {

// Status codes returned through the C ABI (include/bhut_gb300.h).
enum Status : int {
    kOk = 0,
    kInvalid = 1,        // bad argument (maps to ValueError)
    kNotBuilt = 2,       // tree not built
    kCuda = 3,           // CUDA runtime error
    kNoMemory = 4,       // device allocation failed
    kDeviceFlag = 5,     // a kernel raised its error word (stack overflow, ...)
    kInternal = 6,
};

// Error word bits written by kernels (never a trap).
enum DeviceError : unsigned {
    kErrStackOverflow = 1u,
    kErrNonFinite = 2u,
    kErrBadNode = 4u,
    kErrScratchSize = 8u,
};

constexpr int kWarp = 32;
constexpr int kStackDepth = 64;     // per-warp traversal stack entries

void set_error(const char* fmt, ...);
// Counts kernel launches made by the library (reported by bhut_launch_count).
void note_launches(long long k);
int cuda_status(cudaError_t e, const char* what);
// Stream-ordered device memory for the handles' buffers (capi.cu); without
// memory the trees kept for reuse are given back first.
int device_alloc(void** p, size_t bytes, cudaStream_t s);

#define BHUT_CUDA(call)                                              \
    do {                                                             \
        cudaError_t e__ = (call);                                    \
        if (e__ != cudaSuccess) return ::bhut::cuda_status(e__, #call); \
    } while (0)

#define BHUT_TRY(call)                     \
    do {                                   \
        int s__ = (call);                  \
        if (s__ != ::bhut::kOk) return s__; \
    } while (0)

inline unsigned grid_for(int64_t n, int block, unsigned cap = 152u * 16u)
{
    int64_t g = (n + block - 1) / block;
    if (g < 1) g = 1;
    if (g > cap) g = cap;
    return (unsigned)g;
}

// ---------------------------------------------------------------------------
// Radix sort of (uint64 key, int32 value) pairs, stable, LSD, 8-bit digits
// (sort.cu).
// ---------------------------------------------------------------------------
// Keys per tile (sort.cu): more tiles give more blocks for the latency-bound
// rank and scatter steps, at the price of larger count tables.  Whole rebuilds,
// us, by tiles of 256 / 512 / 1,024 / 2,048 keys:
//   32,768   177 / 182 / 208 / 229      300,000    267 / 232 / 238 / 255
//   100,000  205 / 194 / 211 / 236      500,000    350 / 299 / 286 / 288
//   200,000  241 / 220 / 224 / 241      1,000,000  517 / 424 / 395 / 370
#ifndef BHUT_SORT_SMALL_TILE_MAX
#define BHUT_SORT_SMALL_TILE_MAX 320000
#endif
// The fewest keys go without the scan launches: orders of 10,000 / 16,000 /
// 24,000 / 32,768 keys 167 / 173 / 198 / 191 us, with them 201 / 205 / 209 /
// 214 us; rebuilds 167 / 172 / 193 / 185 and 171 / 185 / 185 / 185 us.
#ifndef BHUT_SORT_SUMS_MAX
#define BHUT_SORT_SUMS_MAX 16384
#endif
constexpr int kSortShift = 11, kSortShiftSmall = 9;
constexpr int kSortThreads = 256;
constexpr int kSortPassesMax = 8;      // 64 key bits

constexpr bool sort_small_tiles(int64_t n) { return n <= BHUT_SORT_SMALL_TILE_MAX; }
constexpr bool sort_sums(int64_t n) { return n <= BHUT_SORT_SUMS_MAX; }
constexpr int64_t sort_tiles(int64_t n)
{
    const int shift = sort_small_tiles(n) ? kSortShiftSmall : kSortShift;
    return (n + (1 << shift) - 1) >> shift;
}
constexpr int sort_tables(int64_t n) { return sort_sums(n) ? 3 : 2; }
constexpr size_t sort_align(size_t x) { return (x + 255) & ~(size_t)255; }
// Scratch of radix_sort_pairs for n keys: the ping-pong keys and values, two or
// three count tables (256 x tiles) and the per-pass digit totals.  Not monotone
// in n; largest below a limit L at L itself when L is above both rules' lines.
constexpr size_t sort_scratch_bytes(int64_t n)
{
    return sort_align(sizeof(uint64_t) * (size_t)n) + sort_align(sizeof(int32_t) * (size_t)n) +
           sort_tables(n) * sort_align(sizeof(uint32_t) * 256 * (size_t)sort_tiles(n)) +
           sort_align(sizeof(uint32_t) * 256 * kSortPassesMax);
}
// Sorts keys[0..n) ascending with values carried along.  `bits` is the
// number of low key bits that can be non-zero (passes = ceil(bits / 8)).
// The result ends in keys/vals.  Scratch must hold sort_scratch_bytes(n).
int radix_sort_pairs(uint64_t* keys, int32_t* vals, int64_t n, int bits, void* scratch,
                     cudaStream_t stream);

}  // namespace bhut
