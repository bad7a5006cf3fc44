// Device-wide scan and radix sort primitives (sort.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <stddef.h>

#include "common.cuh"

namespace tdt {

// ------------------------------------------------------------------ look-back
// A tile's status word: its aggregate, then its inclusive prefix, in the low
// bits under two flag bits.  Words are zero before the pass.
template <class S>
struct TileWord {
    static constexpr S kAggregate = S(1) << (8 * sizeof(S) - 2);
    static constexpr S kInclusive = S(2) << (8 * sizeof(S) - 2);
    static constexpr S kValue = kAggregate - 1;
};

// Wait limit of a look-back on a tile that has not published (tiles are handed
// out in order, so the awaited block is running); past it the waiter records
// TDT_ERR_TIMEOUT and goes on with a prefix that is too small, so its results
// stay inside their arrays but leave places unwritten.  Kernels that index by
// such results bound them, or do not start (look_back_failed), and the caller's
// result is rejected.
constexpr uint64_t kLookBackTimeoutNs = 2ull * 1000ull * 1000ull * 1000ull;

struct LookBack {
    int* status;
    unsigned long long limit_ns;
    unsigned clock_mask;         // the clock is read every clock_mask + 1 polls
};
LookBack look_back(int* status);  // with the limit in force (tdt_set_lookback_limit_ns)

// A wait of an earlier kernel ran out.  The same for every thread: where it is
// true no block of the kernel that asks goes on to raise the status.
__device__ __forceinline__ bool look_back_failed(const int* status) {
    return *(const volatile int*)status == (int)TDT_ERR_TIMEOUT;
}

template <class S>
__device__ __forceinline__ S tile_word_wait(const S* p, const LookBack& L) {
    S w = *(const volatile S*)p;
    if (w) return w;
    const uint64_t t0 = globaltimer_ns();
    for (unsigned spins = 1;; spins++) {
        w = *(const volatile S*)p;
        if (w) return w;
        if ((spins & L.clock_mask) == 0 && globaltimer_ns() - t0 > L.limit_ns) {
            atomicMax(L.status, (int)TDT_ERR_TIMEOUT);
            return TileWord<S>::kInclusive;
        }
    }
}

// Sum of the tiles before `tile`, by one whole warp: 32 predecessors at a time
// (words[t] is tile t's).  Lane 0 has published the tile's aggregate.
template <class S>
__device__ __forceinline__ S warp_look_back(const S* words, int64_t tile, const LookBack& L) {
    using W = TileWord<S>;
    S sum = 0;
    for (int64_t t = tile - 1; t >= 0; t -= kWarp) {
        const int64_t mine = t - (int64_t)lane_id();
        const S w = mine >= 0 ? tile_word_wait(words + mine, L) : W::kInclusive;
        const unsigned inc = __ballot_sync(kFull, (w & W::kInclusive) != 0);
        const int last = inc ? __ffs(inc) - 1 : kWarp - 1;  // nearest inclusive prefix
        sum += warp_sum((int)lane_id() <= last ? (S)(w & W::kValue) : S(0));
        if (inc) break;
    }
    return sum;
}

size_t scan_scratch_bytes(int64_t n);
// Scratch is zeroed by the caller; status receives TDT_ERR_TIMEOUT.
// out[i] = sum(in[0..i)), and *total (device, may be null) = sum(in).
int exclusive_scan(const int32_t* in, int64_t* out, int64_t n, int64_t* total, void* scratch, int* status,
                   cudaStream_t st);
// The same over one int32 per vertex (out: nv + 1), and over the staging slots
// of the rows of a CSR (slots: nv + 1; walk.cu).
int scan_rows(const int32_t* in, int64_t* out, void* scratch, const int64_t* rp, int64_t* slots, void* slots_scratch,
              int64_t nv, int* status, cudaStream_t st);
// The same over n > 0 list lengths (out: n + 1), and the choice it leaves: lists
// when their 8-byte entries fit the tail, from the staging slots when they fit
// beside those.
struct ListDecision {
    const int64_t* staged;         // staging slots in all
    unsigned long long tail_bytes;
    const int* stage_skip;         // non-zero: nothing was staged
    int* listed;
    int* list_skip;
    int* compact_skip;
    int* rewalk_skip;
};
int scan_lists(const int32_t* in, int64_t* out, int64_t n, void* scratch, const ListDecision& D, int* status,
               cudaStream_t st);

// ------------------------------------------------------------------ radix sort
// Stable LSD sort by 8-bit digits, one launch per pass: the digit totals of
// every pass come from the kernel that makes the keys (DigitHist), and a tile
// finds where its digits go by looking back over the tiles before it, so a
// pass reads and writes each key once.
constexpr int kRadix = 256;
constexpr int kMaxPasses = 8;

// Scratch of one sort, zeroed by the caller before the key kernel runs.
struct RadixScratch {
    uint32_t* hist;        // [passes][256]
    uint32_t* tile_next;   // [passes]
    void* words;           // [passes][tiles][256]
    size_t bytes;          // of the whole, from hist on
};
RadixScratch radix_scratch(void* base, int64_t n, int passes);  // base may be null (sizes only)

// Digit totals of a key kernel's keys: init, add per key, flush by the block.
struct DigitHist {
    uint32_t* s;           // shared memory, kMaxPasses * kRadix words
    __device__ __forceinline__ void init(int passes) {
        for (int i = threadIdx.x; i < passes * kRadix; i += blockDim.x) s[i] = 0u;
        __syncthreads();
    }
    template <class K>
    __device__ __forceinline__ void add(K key, int passes) {
        for (int p = 0; p < passes; p++) atomicAdd(s + p * kRadix + (unsigned)((key >> (8 * p)) & 0xff), 1u);
    }
    __device__ __forceinline__ void flush(int passes, uint32_t* hist) {
        __syncthreads();
        for (int i = threadIdx.x; i < passes * kRadix; i += blockDim.x)
            if (s[i]) atomicAdd(hist + i, s[i]);
    }
};

// Sorts n keys by their low 8 * passes bits.  in may be another array than the
// two that the passes alternate between (pass 0 writes b0, pass 1 b1, ...); the
// sorted keys are in radix_result.  vals: with kVals the values are the keys'
// indices at first.  n_dev (may be null): the number of keys, at most n, read on
// the device.  max_dev (may be null): passes above the highest set digit of
// *max_dev do nothing, and the result is in the buffer of the last pass that
// ran (radix_passes_run).
template <class K, bool kVals>
int radix_sort(const K* in, K* b0, K* b1, uint32_t* v0, uint32_t* v1, int64_t n, int passes, const RadixScratch& R,
               const uint32_t* n_dev, const long long* max_dev, int* status, cudaStream_t st);

__host__ __device__ inline int radix_passes_run(int passes, long long max_key) {
    int p = 1;
    while (p < passes && (max_key >> (8 * p)) != 0) p++;
    return p;
}

}  // namespace tdt
