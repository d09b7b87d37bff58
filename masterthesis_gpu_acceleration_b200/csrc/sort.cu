// sort.cu — radix sort of 64-bit keys (the index build) and, from its passes,
// distinct-pair counting (the sort mode of the body-size deduplication).
//
// In sort mode the engine appends one 64-bit key per body grounding that
// reaches hO: [sort index of the plan | hS row | hO rank] (see emit_pair in
// kernels.cu).  Equal keys only have to meet, not to be in order: one or two
// radix passes over a hash of the keys (8 bits a pass) part them into buckets
// of a few thousand, and a block counts each bucket's distinct keys per plan
// through a hash set in shared memory.  (Sorting all 41 bits in use took six
// passes and 25 launches: a call with 1.3M keys takes 0.63 ms on the device
// now, 0.79 ms then.)  The
// reference does the same job with Thrust: a comparison sort of int2 pairs
// followed by unique (GPU_03/gpu_rules_lib.cu:485-518, after an
// overflow-and-double retry loop); here the buffer is sized exactly from the
// append cursor when an estimate was short (see Staged in engine.hpp).
//
// Per pass (tile = 2,048 keys, 256 threads x 8 keys, read coalesced):
//   radix_hist_kernel     digit counts per tile, stored digit-major, and
//                         per-digit totals
//   radix_scan_kernel     one block per digit: the exclusive prefix of its
//                         counts over tiles, plus the digit's base
//   radix_scatter_kernel  stable rank of each key within its tile
//                         (__match_any_sync per warp, then a prefix over
//                         (key round, warp) per digit), keys reordered by
//                         digit in shared memory and written out in runs
// The key count lives on the device (the append cursor, clamped to the
// capacity), so every kernel reads it there and the whole sequence can be
// captured in a CUDA graph with grids sized for the capacity.
#include <cuda_runtime.h>

#include <cstdint>

#include "common.hpp"

namespace gr {
namespace {

constexpr int kSortThreads = 256;
constexpr int kSortPerThread = 8;
constexpr int kSortTile = kSortThreads * kSortPerThread;
constexpr int kRadix = 256;
constexpr int kSortWarps = kSortThreads / 32;

__device__ __forceinline__ long long keys_in(const unsigned long long* count, unsigned long long cap) {
    const unsigned long long n = *count;
    return (long long)(n < cap ? n : cap);
}

// The digit of a key at `shift`: of its own bits, or (kHash) of a hash of them.
__device__ __forceinline__ uint32_t key_hash(unsigned long long x) {
    x ^= x >> 29;
    x *= 0x9E3779B97F4A7C15ull;
    return (uint32_t)(x >> 32);
}
// A second mix, one to one over 64 bits.
__device__ __forceinline__ unsigned long long key_mix(unsigned long long x) {
    x ^= x >> 32;
    return x * 0xA24BAED4963EE407ull;
}
template <bool kHash>
__device__ __forceinline__ int key_digit(unsigned long long x, int shift) {
    if constexpr (kHash) return (int)((key_hash(x) >> shift) & (kRadix - 1));
    else return (int)((unsigned)(x >> shift) & (kRadix - 1));
}

// hist[d * tilesCap + t]: keys of tile t with digit d; hist[kRadix * tilesCap + d]:
// keys with digit d (zeroed before the pass).
template <bool kHash>
__global__ void __launch_bounds__(kSortThreads)
radix_hist_kernel(const unsigned long long* __restrict__ keys, const unsigned long long* count, unsigned long long cap,
                  int shift, uint32_t* hist, long long tilesCap) {
    __shared__ uint32_t h[kRadix];
    const long long n = keys_in(count, cap);
    const long long tiles = (n + kSortTile - 1) / kSortTile;
    uint32_t* totals = hist + (size_t)kRadix * tilesCap;
    for (long long t = blockIdx.x; t < tiles; t += gridDim.x) {
        h[threadIdx.x] = 0u;
        __syncthreads();
        const long long base = t * kSortTile;
        const unsigned lower = (1u << (threadIdx.x & 31)) - 1u;
#pragma unroll
        for (int k = 0; k < kSortPerThread; ++k) {
            const long long i = base + (long long)k * kSortThreads + threadIdx.x;
            const int d = i < n ? key_digit<kHash>(keys[i], shift) : kRadix;
            // one shared atomic per distinct digit of the warp (the high
            // digits of small keys are mostly equal)
            const unsigned peers = __match_any_sync(0xffffffffu, d);
            if (d < kRadix && (peers & lower) == 0) atomicAdd(&h[d], (uint32_t)__popc(peers));
        }
        __syncthreads();
        const uint32_t c = h[threadIdx.x];
        hist[(size_t)threadIdx.x * tilesCap + t] = c;
        if (c) atomicAdd(&totals[threadIdx.x], c);
        __syncthreads();
    }
}

// Block-wide inclusive scan of one value per thread (blockDim.x = 1024).
__device__ __forceinline__ uint32_t block_incl_scan(uint32_t v, uint32_t* warpSums) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, v, d);
        if (lane >= d) v += y;
    }
    if (lane == 31) warpSums[warp] = v;
    __syncthreads();
    if (warp == 0) {
        const int nw = blockDim.x >> 5;
        uint32_t w = lane < nw ? warpSums[lane] : 0u;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, w, d);
            if (lane >= d) w += y;
        }
        if (lane < nw) warpSums[lane] = w;
    }
    __syncthreads();
    return v + (warp > 0 ? warpSums[warp - 1] : 0u);
}

// One block per digit d: hist[d][t] becomes the output position of tile t's
// first key with digit d.
__global__ void __launch_bounds__(1024)
radix_scan_kernel(uint32_t* hist, const unsigned long long* count, unsigned long long cap, long long tilesCap) {
    __shared__ uint32_t warpSums[32];
    __shared__ uint32_t base;
    const int d = blockIdx.x;
    const long long n = keys_in(count, cap);
    const long long tiles = (n + kSortTile - 1) / kSortTile;
    const uint32_t* totals = hist + (size_t)kRadix * tilesCap;
    if (threadIdx.x < 32) {
        uint32_t b = 0;
        for (int e = (int)threadIdx.x; e < d; e += 32) b += totals[e];
#pragma unroll
        for (int o = 16; o; o >>= 1) b += __shfl_xor_sync(0xffffffffu, b, o);
        if (threadIdx.x == 0) base = b;
    }
    __syncthreads();
    uint32_t carry = base;
    uint32_t* row = hist + (size_t)d * tilesCap;
    for (long long c0 = 0; c0 < tiles; c0 += blockDim.x) {
        const long long i = c0 + threadIdx.x;
        const uint32_t v = i < tiles ? row[i] : 0u;
        const uint32_t incl = block_incl_scan(v, warpSums);
        if (i < tiles) row[i] = carry + incl - v;
        // every thread reads the chunk's total before the next chunk's scan
        // overwrites warpSums
        carry += warpSums[(blockDim.x >> 5) - 1];
        __syncthreads();
    }
}

template <bool kHash>
__global__ void __launch_bounds__(kSortThreads)
radix_scatter_kernel(const unsigned long long* __restrict__ in, unsigned long long* __restrict__ out,
                     const unsigned long long* count, unsigned long long cap, int shift, const uint32_t* hist,
                     long long tilesCap) {
    // per (key round k, warp w, digit d): keys of that warp and round with
    // digit d, then their exclusive prefix in tile order; the same memory
    // later holds the tile reordered by digit
    __shared__ union {
        uint16_t cnt[kSortPerThread][kSortWarps][kRadix];
        unsigned long long tile[kSortTile];
    } sh;
    __shared__ uint32_t dStart[kRadix];   // tile-local first position of each digit
    __shared__ uint32_t dOut[kRadix];     // output position of the tile's first key of each digit
    __shared__ uint32_t warpSums[kSortWarps];
    const long long n = keys_in(count, cap);
    const long long tiles = (n + kSortTile - 1) / kSortTile;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned lower = (1u << lane) - 1u;
    for (long long t = blockIdx.x; t < tiles; t += gridDim.x) {
        uint32_t* c32 = reinterpret_cast<uint32_t*>(&sh.cnt[0][0][0]);
        for (int i = tid; i < kSortPerThread * kSortWarps * kRadix / 2; i += kSortThreads) c32[i] = 0u;
        __syncthreads();
        const long long base = t * kSortTile;
        unsigned long long key[kSortPerThread];
        int dig[kSortPerThread];
        int below[kSortPerThread];
#pragma unroll
        for (int k = 0; k < kSortPerThread; ++k) {
            const long long i = base + (long long)k * kSortThreads + tid;
            key[k] = i < n ? in[i] : 0ull;
            dig[k] = i < n ? key_digit<kHash>(key[k], shift) : kRadix;
            const unsigned peers = __match_any_sync(0xffffffffu, dig[k]);
            below[k] = __popc(peers & lower);
            if (dig[k] < kRadix && below[k] == 0) sh.cnt[k][warp][dig[k]] = (uint16_t)__popc(peers);
        }
        __syncthreads();
        // thread d: prefix of digit d over (round, warp), i.e. in tile order
        uint32_t run = 0;
        for (int k = 0; k < kSortPerThread; ++k)
            for (int w = 0; w < kSortWarps; ++w) {
                const uint32_t x = sh.cnt[k][w][tid];
                sh.cnt[k][w][tid] = (uint16_t)run;
                run += x;
            }
        dOut[tid] = hist[(size_t)tid * tilesCap + t];
        // exclusive scan of the per-digit tile counts over the 256 digits
        uint32_t v = run;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, v, d);
            if (lane >= d) v += y;
        }
        if (lane == 31) warpSums[warp] = v;
        __syncthreads();
        uint32_t before = 0;
        for (int w = 0; w < warp; ++w) before += warpSums[w];
        dStart[tid] = before + v - run;
        __syncthreads();
        uint32_t pos[kSortPerThread];
#pragma unroll
        for (int k = 0; k < kSortPerThread; ++k)
            pos[k] = dig[k] < kRadix ? dStart[dig[k]] + sh.cnt[k][warp][dig[k]] + (uint32_t)below[k] : 0xffffffffu;
        __syncthreads();   // the counters are read; the tile may overwrite them
#pragma unroll
        for (int k = 0; k < kSortPerThread; ++k)
            if (pos[k] != 0xffffffffu) sh.tile[pos[k]] = key[k];
        __syncthreads();
        const int m = (int)(n - base < kSortTile ? n - base : kSortTile);
        for (int j = tid; j < m; j += kSortThreads) {
            const unsigned long long x = sh.tile[j];
            const int d = key_digit<kHash>(x, shift);
            out[(size_t)dOut[d] + (size_t)(j - (int)dStart[d])] = x;
        }
        __syncthreads();
    }
}

// Distinct keys per plan of the bucketed keys (grouped by the low 8 x passes
// bits of their hash), added to the plans' results: the key's bits from
// slotShift up are the plan's sort index, slotOf maps it to a result slot.  A
// block takes a run of buckets with about kPartKeys keys (found by binary
// search) and inserts them into a hash set in shared memory; duplicates cost a
// look-up each, wherever they stand.  A part with more distinct keys than the set may hold is taken in
// halves, quarters ... by the leading bits of a second, reversible mix of the
// key, so that every split ends.  A sort index outside [0, nSlots) is reported
// through status (bit 64) and skipped.
constexpr int kSetBits = 13;
constexpr int kSet = 1 << kSetBits;            // entries (64 KB)
static_assert(kSortSetKeys + kSortThreads < kSet, "each thread may insert one more key into a full set");
constexpr int kSlotCounters = 64;              // plans counted in shared memory first
constexpr int kPartKeys = 4096;                // keys of a part, on average
constexpr int kBucketKeys = 5632;              // most keys a bucket should hold, on average
constexpr unsigned long long kNoKey = ~0ull;   // (a key of all ones is counted by itself)

__global__ void __launch_bounds__(kSortThreads)
pairs_distinct_kernel(const unsigned long long* __restrict__ keys, const unsigned long long* count,
                      unsigned long long cap, int passes, int slotShift, const int32_t* slotOf, int nSlots,
                      unsigned long long* results, int* status, int setKeys) {
    extern __shared__ unsigned long long set[];
    __shared__ unsigned counters[kSlotCounters];
    __shared__ int held, ones;
    __shared__ long long range[2];
    const long long n = keys_in(count, cap);
    const long long nb = 1ll << (8 * passes);
    const uint32_t mask = (uint32_t)nb - 1u;
    const long long parts = min(nb, (n + kPartKeys - 1) / kPartKeys);
    const int tid = threadIdx.x;
    auto add = [&](unsigned long long x) {
        const unsigned long long s = x >> slotShift;
        if (s >= (unsigned long long)nSlots) atomicOr(status, 64);
        else if (s < kSlotCounters) atomicAdd(&counters[s], 1u);
        else atomicAdd(results + slotOf[s], 1ull);
    };
    for (long long b = blockIdx.x; b < parts; b += gridDim.x) {
        if (tid < 64) {   // first key of part b, and of the one after it: a warp each, 32 pivots a step
            const int lane = tid & 31;
            const uint32_t target = (uint32_t)((b + (tid >> 5)) * nb / parts);
            long long lo = 0, hi = n;
            while (lo < hi) {
                const long long len = hi - lo;
                const long long at = len <= 32 ? lo + lane : lo + len * (lane + 1) / 33;
                const bool below = at < hi && (key_hash(keys[at]) & mask) < target;
                const int c = __popc(__ballot_sync(0xffffffffu, below));   // (the first c pivots are below)
                if (len <= 32) {
                    lo += c;
                    break;
                }
                const long long from = c > 0 ? lo + len * c / 33 + 1 : lo;
                hi = c < 32 ? lo + len * (c + 1) / 33 : hi;
                lo = from;
            }
            if (lane == 0) range[tid >> 5] = lo;
        }
        __syncthreads();
        const long long beg = range[0], end = range[1];
        if (tid < kSlotCounters) counters[tid] = 0u;
        // the keys whose mix starts with the r bits v; a set that overflows is
        // taken as its two halves (at 52 bits fewer than 4,096 keys are left)
        unsigned long long v = 0;
        for (int r = 0; beg < end;) {
            for (int i = tid; i < kSet; i += kSortThreads) set[i] = kNoKey;
            if (tid == 0) held = ones = 0;
            __syncthreads();
            for (long long i = beg + tid; i < end; i += kSortThreads) {
                const unsigned long long x = keys[i];
                if (r > 0 && key_mix(x) >> (64 - r) != v) continue;
                if (x == kNoKey) { ones = 1; continue; }
                unsigned at = (unsigned)(x * 0xD6E8FEB86659FD93ull >> (64 - kSetBits));
                for (int probe = 0; probe < kSet; ++probe) {
                    const unsigned long long old = *(volatile unsigned long long*)&set[at];
                    if (old == x) break;
                    if (old == kNoKey) {
                        if (*(volatile int*)&held >= setKeys) break;   // full: seen after the barrier
                        const unsigned long long seen = atomicCAS(&set[at], kNoKey, x);
                        if (seen == x) break;
                        if (seen == kNoKey) { atomicAdd(&held, 1); break; }
                    }
                    at = (at + 1) & (kSet - 1);
                }
            }
            __syncthreads();
            const bool full = held >= setKeys;
            if (full) {
                ++r;
                v <<= 1;
                __syncthreads();   // `held` is read
                continue;
            }
            for (int i = tid; i < kSet; i += kSortThreads)
                if (set[i] != kNoKey) add(set[i]);
            if (tid == 0 && ones) add(kNoKey);
            while (r > 0 && (v & 1)) {   // both halves done
                v >>= 1;
                --r;
            }
            if (r == 0) break;
            ++v;
            __syncthreads();   // the set is read
        }
        __syncthreads();
        for (int i = tid; i < kSlotCounters && i < nSlots; i += kSortThreads)
            if (counters[i]) atomicAdd(results + slotOf[i], (unsigned long long)counters[i]);
        __syncthreads();
    }
}

}  // namespace

size_t pairs_sort_hist_words(unsigned long long cap) {
    const unsigned long long tiles = (cap + kSortTile - 1) / kSortTile;
    return (size_t)kRadix * (size_t)(tiles > 0 ? tiles : 1) + kRadix;
}

unsigned long long* radix_sort_keys(unsigned long long* keys, unsigned long long* tmp, const unsigned long long* count,
                                    unsigned long long cap, int bits, uint32_t* hist, int grid, cudaStream_t stream,
                                    cudaError_t* err);

template <bool kHash>
static unsigned long long* radix_passes(unsigned long long* keys, unsigned long long* tmp,
                                        const unsigned long long* count, unsigned long long cap, int bits,
                                        uint32_t* hist, int grid, cudaStream_t stream, cudaError_t* err);

int pairs_sort_passes(unsigned long long cap) {
    int p = 1;
    while (p < 3 && cap > ((unsigned long long)kBucketKeys << (8 * p))) ++p;
    return p;
}

// Groups the first min(*count, cap) keys by a hash, ping-ponging between keys
// and tmp, and adds each plan's distinct keys to results[slotOf[key >>
// slotShift]] (nSlots sort indices; status as the engine's).  hist:
// pairs_sort_hist_words(cap) words.  grid: blocks of the per-tile kernels
// (they loop over tiles).  setKeys: most keys a hash set takes in one round.
cudaError_t pairs_sort_count(unsigned long long* keys, unsigned long long* tmp, const unsigned long long* count,
                             unsigned long long cap, int slotShift, const int32_t* slotOf, int nSlots,
                             unsigned long long* results, int* status, uint32_t* hist, int grid, int setKeys,
                             cudaStream_t stream) {
    if (cap == 0) return cudaSuccess;
    if (slotShift < 0 || slotShift > 63 || cap > 0xffffffffull) return cudaErrorInvalidValue;
    cudaError_t e = cudaSuccess;
    const int passes = pairs_sort_passes(cap);
    unsigned long long* a = radix_passes<true>(keys, tmp, count, cap, 8 * passes, hist, grid, stream, &e);
    if (e != cudaSuccess) return e;
    const size_t smem = sizeof(unsigned long long) * kSet;
    e = cudaFuncSetAttribute(pairs_distinct_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    const long long parts = (long long)((cap + kPartKeys - 1) / kPartKeys);
    pairs_distinct_kernel<<<(int)(parts < grid ? parts : grid), kSortThreads, smem, stream>>>(
        a, count, cap, passes, slotShift, slotOf, nSlots, results, status, setKeys);
    return cudaGetLastError();
}

unsigned long long* radix_sort_keys(unsigned long long* keys, unsigned long long* tmp, const unsigned long long* count,
                                    unsigned long long cap, int bits, uint32_t* hist, int grid, cudaStream_t stream,
                                    cudaError_t* err) {
    *err = cudaSuccess;
    if (cap == 0) return keys;
    if (bits < 1 || bits > 64 || cap > 0xffffffffull) {
        *err = cudaErrorInvalidValue;
        return keys;
    }
    return radix_passes<false>(keys, tmp, count, cap, bits, hist, grid, stream, err);
}

template <bool kHash>
static unsigned long long* radix_passes(unsigned long long* keys, unsigned long long* tmp,
                                        const unsigned long long* count, unsigned long long cap, int bits,
                                        uint32_t* hist, int grid, cudaStream_t stream, cudaError_t* err) {
    *err = cudaSuccess;
    const long long tilesCap = (long long)((cap + kSortTile - 1) / kSortTile);
    const int g = (int)(tilesCap < grid ? tilesCap : grid);
    unsigned long long* a = keys;
    unsigned long long* b = tmp;
    for (int shift = 0; shift < bits; shift += 8) {
        cudaError_t e = cudaMemsetAsync(hist + (size_t)kRadix * tilesCap, 0, kRadix * sizeof(uint32_t), stream);
        if (e != cudaSuccess) { *err = e; return a; }
        radix_hist_kernel<kHash><<<g, kSortThreads, 0, stream>>>(a, count, cap, shift, hist, tilesCap);
        radix_scan_kernel<<<kRadix, 1024, 0, stream>>>(hist, count, cap, tilesCap);
        radix_scatter_kernel<kHash><<<g, kSortThreads, 0, stream>>>(a, b, count, cap, shift, hist, tilesCap);
        unsigned long long* x = a;
        a = b;
        b = x;
    }
    *err = cudaGetLastError();
    return a;
}

}  // namespace gr
