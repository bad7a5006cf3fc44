// Device-wide exclusive scan and stable LSD radix sort (8-bit digits).
//
// Both are single-pass: a tile publishes its totals and finds its start by
// looking back over the tiles before it (tiles are handed out in order, so the
// tiles waited for are running).  The scan is one launch instead of three; a
// sort pass is one launch instead of five, and reads its keys once instead of
// twice, with no digit table of all tiles to scan between.  The methods are
// published: the scan with look-back by Merrill and Garland (Single-pass Parallel
// Prefix Scan with Decoupled Look-back, 2016), the sort by Adinets and Merrill
// (Onesweep: A Faster Least Significant Digit Radix Sort for GPUs, 2022).  A pass over 67 M
// 64-bit keys: 600 -> 400 us, 350 with the ballots below (bound: 16 bytes a
// key, 160 us).
#include "sort.cuh"

namespace tdt {

// Test knob: wait limit of the look-backs launched next (<= 0: the default).
static long long g_look_back_limit_ns = 0;
void set_look_back_limit(long long ns) { g_look_back_limit_ns = ns; }
LookBack look_back(int* status) {
    if (g_look_back_limit_ns > 0) return {status, (unsigned long long)g_look_back_limit_ns, 0u};
    return {status, kLookBackTimeoutNs, 63u};
}

constexpr int kScanBlock = 512;
constexpr int kScanItems = 8;
constexpr int kScanTile = kScanBlock * kScanItems;

template <class T>
__device__ __forceinline__ T block_excl_scan(T v, T* s_warp, T* total) {
    const unsigned lane = lane_id();
    const int w = threadIdx.x / kWarp;
    T incl = warp_incl_scan(v);
    if (lane == 31) s_warp[w] = incl;
    __syncthreads();
    if (w == 0) {
        T x = (lane < blockDim.x / kWarp) ? s_warp[lane] : T(0);
        T xi = warp_incl_scan(x);
        if (lane < blockDim.x / kWarp) s_warp[lane] = xi - x;
        if (lane == 31) s_warp[32] = xi;
    }
    __syncthreads();
    T res = s_warp[w] + incl - v;
    if (total) *total = s_warp[32];
    __syncthreads();
    return res;
}

// What a scan adds up.
template <class TI>
struct ScanArray {
    const TI* in;
    __device__ __forceinline__ int64_t operator()(int64_t i) const { return (int64_t)in[i]; }
};
// Staging slots of row i of a CSR (d (d - 1) / 2 for d entries; 0 once an error
// is known).
struct ScanStageSlots {
    const int64_t* rp;
    const int* status;
    __device__ __forceinline__ int64_t operator()(int64_t i) const {
        const int64_t d = rp[i + 1] - rp[i];
        return *(volatile const int*)status == 0 && d > 1 ? d * (d - 1) / 2 : 0;
    }
};

template <class In>
struct ScanJob {
    In in;
    int64_t n;
    int64_t* out;
    int64_t* total;
    unsigned long long* words;
    unsigned* next;
    int64_t tiles;
};

// One tile of a job; done(total) is called by one thread of the last tile.
template <class In, class Done>
__device__ __forceinline__ void scan_tile(const ScanJob<In>& J, const LookBack& L, Done&& done) {
    using W = TileWord<unsigned long long>;
    using TO = int64_t;
    __shared__ TO s_warp[33];
    __shared__ unsigned s_tile;
    __shared__ unsigned long long s_before;
    if (threadIdx.x == 0) s_tile = atomicAdd(J.next, 1u);
    __syncthreads();
    const int64_t tile = s_tile, n = J.n;
    const int64_t base = tile * kScanTile + (int64_t)threadIdx.x * kScanItems;
    TO v[kScanItems];
    TO sum = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; k++) {
        v[k] = base + k < n ? J.in(base + k) : TO(0);
        sum += v[k];
    }
    TO tot;
    TO run = block_excl_scan<TO>(sum, s_warp, &tot);
    if (threadIdx.x < kWarp) {
        if (threadIdx.x == 0)
            *(volatile unsigned long long*)(J.words + tile) =
                (tile == 0 ? W::kInclusive : W::kAggregate) | (unsigned long long)tot;
        const unsigned long long before = warp_look_back(J.words, tile, L);
        if (threadIdx.x == 0) {
            if (tile > 0)
                *(volatile unsigned long long*)(J.words + tile) =
                    W::kInclusive | ((before + (unsigned long long)tot) & W::kValue);
            s_before = before;
        }
    }
    __syncthreads();
    run += (TO)s_before;
#pragma unroll
    for (int k = 0; k < kScanItems; k++) {
        if (base + k < n) J.out[base + k] = run;
        run += v[k];
    }
    if (tile == J.tiles - 1 && threadIdx.x == kScanBlock - 1) {
        if (J.total) *J.total = run;
        done(run);
    }
}

__global__ void __launch_bounds__(kScanBlock) scan_kernel(ScanJob<ScanArray<int32_t>> J, LookBack L) {
    scan_tile(J, L, [](int64_t) {});
}

// The in-adjacency's offsets and the rows' staging slots, tiles of both in one
// launch (a launch and 5 us of a small call).
__global__ void __launch_bounds__(kScanBlock) scan_rows_kernel(ScanJob<ScanArray<int32_t>> J,
                                                               ScanJob<ScanStageSlots> K, LookBack L) {
    if (blockIdx.x < J.tiles) scan_tile(J, L, [](int64_t) {});
    else scan_tile(K, L, [](int64_t) {});
}

// The lists' offsets, and whether there are lists.
__global__ void __launch_bounds__(kScanBlock) scan_lists_kernel(ScanJob<ScanArray<int32_t>> J, ListDecision D,
                                                                LookBack L) {
    scan_tile(J, L, [&](int64_t need) {
        const unsigned long long slots = D.tail_bytes / 8;
        const int ok = *(volatile int*)L.status == 0 && (unsigned long long)need <= slots;
        const int compact = ok && !*D.stage_skip && (unsigned long long)need <= slots - (unsigned long long)*D.staged;
        *D.listed = ok;
        *D.list_skip = !ok;
        *D.compact_skip = !compact;
        *D.rewalk_skip = !ok || compact;
    });
}

size_t scan_scratch_bytes(int64_t n) {
    const int64_t nb = (n + kScanTile - 1) / kScanTile;
    return (size_t)(nb + 1) * 8 + 256;
}

template <class In>
static ScanJob<In> scan_job(In in, int64_t* out, int64_t n, int64_t* total, void* scratch) {
    const int64_t nb = (n + kScanTile - 1) / kScanTile;
    unsigned long long* words = reinterpret_cast<unsigned long long*>(scratch);
    return {in, n, out, total, words, reinterpret_cast<unsigned*>(words + nb), nb};
}

int exclusive_scan(const int32_t* in, int64_t* out, int64_t n, int64_t* total, void* scratch, int* status,
                   cudaStream_t st) {
    if (n <= 0) {
        if (total) TDT_CUDA(cudaMemsetAsync(total, 0, sizeof(int64_t), st));
        return TDT_OK;
    }
    const auto J = scan_job(ScanArray<int32_t>{in}, out, n, total, scratch);
    scan_kernel<<<(unsigned)J.tiles, kScanBlock, 0, st>>>(J, look_back(status));
    TDT_LAUNCH_CHECK("scan");
    return TDT_OK;
}

int scan_rows(const int32_t* in, int64_t* out, void* scratch, const int64_t* rp, int64_t* slots, void* slots_scratch,
              int64_t nv, int* status, cudaStream_t st) {
    if (nv <= 0) {
        TDT_CUDA(cudaMemsetAsync(out, 0, sizeof(int64_t), st));
        TDT_CUDA(cudaMemsetAsync(slots, 0, sizeof(int64_t), st));
        return TDT_OK;
    }
    const auto J = scan_job(ScanArray<int32_t>{in}, out, nv, out + nv, scratch);
    const auto K = scan_job(ScanStageSlots{rp, status}, slots, nv, slots + nv, slots_scratch);
    scan_rows_kernel<<<(unsigned)(J.tiles + K.tiles), kScanBlock, 0, st>>>(J, K, look_back(status));
    TDT_LAUNCH_CHECK("scan_rows");
    return TDT_OK;
}

int scan_lists(const int32_t* in, int64_t* out, int64_t n, void* scratch, const ListDecision& D, int* status,
               cudaStream_t st) {
    TDT_CHECK_ARG(n > 0, "no lists");
    const auto J = scan_job(ScanArray<int32_t>{in}, out, n, out + n, scratch);
    scan_lists_kernel<<<(unsigned)J.tiles, kScanBlock, 0, st>>>(J, D, look_back(status));
    TDT_LAUNCH_CHECK("scan_lists");
    return TDT_OK;
}

// ------------------------------------------------------------------ radix sort
constexpr int kSortBlock = 256;   // one thread per digit
constexpr int kSortWarps = kSortBlock / kWarp;
static_assert(kSortBlock == kRadix, "one thread per digit");
// Keys per thread: 16 leave four blocks per SM, long runs of a digit and few
// look-backs; a sort of few tiles is a chain of latencies, so its tiles are
// smaller (65,536 / 0.8 M / 67 M draws preprocessed: 318 us / 390 us / 6.77 ms
// with 12, 326 / 406 / 6.26 with 16, 24 at three blocks per SM 332 us / 6.17 ms).
constexpr int kSortItems = 16, kSortSmallItems = 12;
constexpr int64_t kSortSmall = 1 << 20;
constexpr int kSortBatch = 4;          // steps ranked together
static_assert(kSortItems % kSortBatch == 0 && kSortSmallItems % kSortBatch == 0, "whole batches");
constexpr int kBack = 4;               // tiles looked back on at a time
static int64_t sort_tile(int64_t n) { return (int64_t)kSortBlock * (n < kSortSmall ? kSortSmallItems : kSortItems); }
// counts fit 30 bits below this many keys
constexpr int64_t kWideKeys = 1ll << 30;

template <class K, class S, bool kVals, bool kIota, int kItems>
__global__ void __launch_bounds__(kSortBlock, 4) radix_pass_kernel(
    const K* __restrict__ keys_in, const uint32_t* __restrict__ vals_in, K* __restrict__ keys_out,
    uint32_t* __restrict__ vals_out, int64_t n, int pass, const uint32_t* __restrict__ hist,
    uint32_t* tile_next, S* words, const uint32_t* n_dev, const long long* max_dev, LookBack L) {
    using W = TileWord<S>;
    constexpr int kTile = kSortBlock * kItems;
    if (max_dev && pass > 0 && (*max_dev >> (8 * pass)) == 0) return;
    if (n_dev) n = *n_dev < n ? (int64_t)*n_dev : n;
    extern __shared__ __align__(16) unsigned char smem[];
    K* s_keys = reinterpret_cast<K*>(smem);
    uint32_t* s_vals = reinterpret_cast<uint32_t*>(smem + sizeof(K) * kTile);
    __shared__ uint32_t s_wcnt[kSortWarps][kRadix];  // per warp: counts, then first places in the tile
    __shared__ uint32_t s_to[kRadix];      // first place of the digit in the output minus that in the tile (mod 2^32)
    __shared__ uint32_t s_tmp[33];
    __shared__ unsigned s_tile;
    const int w = threadIdx.x / kWarp;
    const unsigned lane = lane_id();
    const int shift = 8 * pass;
    if (threadIdx.x == 0) s_tile = atomicAdd(tile_next, 1u);
    for (int i = lane; i < kRadix; i += kWarp) s_wcnt[w][i] = 0;
    __syncthreads();
    const int64_t tile = s_tile;
    const int64_t base = tile * kTile;
    if (base >= n) return;
    // warp w owns the contiguous sub-tile of kItems * 32 keys; ranks among
    // its keys of the same digit
    K key[kItems];
    uint32_t val[kVals ? kItems : 1];
    uint16_t rank[kItems];
    const int64_t mine = base + (int64_t)w * (kItems * kWarp) + lane;
#pragma unroll
    for (int it = 0; it < kItems; it++) {
        const int64_t i = mine + it * kWarp;
        key[it] = i < n ? keys_in[i] : ~K(0);
        if (kVals) val[it] = kIota ? (uint32_t)i : (i < n ? vals_in[i] : 0u);
    }
    // The first lane of a step's equal digits counts them in the warp's row, and
    // all of them rank from its result, kSortBatch steps at a time.  The equal
    // digits come from eight ballots: __match_any_sync takes a turn per distinct
    // value and held the passes over random digits at 0.58 ms, over skewed ones at
    // 0.36 (67 M keys; preprocessing 7.70 -> 6.77 ms with the ballots, 6.97 with
    // lane masks OR-ed in shared memory).  Keys past the end have the last digit
    // and the last places, which are not written.
#pragma unroll
    for (int b0 = 0; b0 < kItems; b0 += kSortBatch) {
        unsigned peers[kSortBatch];
        uint32_t pre[kSortBatch];
#pragma unroll
        for (int j = 0; j < kSortBatch; j++) {
            const unsigned d = (unsigned)((key[b0 + j] >> shift) & 0xff);
            peers[j] = kFull;
#pragma unroll
            for (int b = 0; b < 8; b++) {
                const bool p = (d >> b) & 1u;
                const unsigned v = __ballot_sync(kFull, p);
                peers[j] &= p ? v : ~v;
            }
        }
#pragma unroll
        for (int j = 0; j < kSortBatch; j++) {
            const unsigned d = (unsigned)((key[b0 + j] >> shift) & 0xff);
            pre[j] = 0;
            if ((peers[j] & lanemask_lt()) == 0) pre[j] = atomicAdd(&s_wcnt[w][d], (uint32_t)__popc(peers[j]));
            __syncwarp();
        }
#pragma unroll
        for (int j = 0; j < kSortBatch; j++)
            rank[b0 + j] = (uint16_t)(__shfl_sync(kFull, pre[j], __ffs(peers[j]) - 1) + __popc(peers[j] & lanemask_lt()));
    }
    __syncthreads();
    const int d = threadIdx.x;
    uint32_t cnt = 0;
#pragma unroll
    for (int ww = 0; ww < kSortWarps; ww++) cnt += s_wcnt[ww][d];
    S* mine_w = words + tile * kRadix + d;
    *(volatile S*)mine_w = (tile == 0 ? W::kInclusive : W::kAggregate) | (S)cnt;
    // the digit's first place in the tile, for each warp, and in the output
    const uint32_t start = block_excl_scan<uint32_t>(cnt, s_tmp, nullptr);
    uint32_t run = start;
#pragma unroll
    for (int ww = 0; ww < kSortWarps; ww++) {
        const uint32_t c = s_wcnt[ww][d];
        s_wcnt[ww][d] = run;
        run += c;
    }
    const uint32_t digit0 = block_excl_scan<uint32_t>(__ldg(hist + d), s_tmp, nullptr);
#pragma unroll
    for (int it = 0; it < kItems; it++) {
        const uint32_t p = s_wcnt[w][(unsigned)((key[it] >> shift) & 0xff)] + rank[it];
        s_keys[p] = key[it];
        if (kVals) s_vals[p] = val[it];
    }
    S before = 0;
    if (tile > 0) {
        // the rows of words of the tiles before, kBack of them in flight
        bool more = true;
        for (int64_t t = tile - 1; more && t >= 0; t -= kBack) {
            S x[kBack];
#pragma unroll
            for (int j = 0; j < kBack; j++) x[j] = t - j >= 0 ? *(const volatile S*)(words + (t - j) * kRadix + d) : S(0);
#pragma unroll
            for (int j = 0; j < kBack; j++) {
                if (!more || t - j < 0) continue;
                if (x[j] == 0) x[j] = tile_word_wait(words + (t - j) * kRadix + d, L);
                before += x[j] & W::kValue;
                more = (x[j] & W::kInclusive) == 0;
            }
        }
        *(volatile S*)mine_w = W::kInclusive | ((before + (S)cnt) & W::kValue);
    }
    s_to[d] = digit0 + (uint32_t)before - start;
    __syncthreads();
    const int tile_n = (int)(n - base < kTile ? n - base : kTile);
    for (int i = threadIdx.x; i < tile_n; i += kSortBlock) {
        const K k = s_keys[i];
        const uint32_t g = s_to[(unsigned)((k >> shift) & 0xff)] + (uint32_t)i;
        if (g < n) {
            keys_out[g] = k;
            if (kVals) vals_out[g] = s_vals[i];
        }
    }
}

RadixScratch radix_scratch(void* base, int64_t n, int passes) {
    const size_t ntiles = (size_t)((n + sort_tile(n) - 1) / sort_tile(n));
    const size_t head = ((size_t)kMaxPasses * kRadix + kMaxPasses) * 4 + 224;  // a multiple of 256
    const size_t word = n < kWideKeys ? 4 : 8;
    RadixScratch R;
    R.hist = reinterpret_cast<uint32_t*>(base);
    R.tile_next = base ? R.hist + kMaxPasses * kRadix : nullptr;
    R.words = base ? (void*)(reinterpret_cast<char*>(base) + head) : nullptr;
    R.bytes = head + (size_t)passes * ntiles * kRadix * word;
    return R;
}

template <class K, class S, bool kVals, int kItems>
static int radix_passes(const K* in, K* b0, K* b1, uint32_t* v0, uint32_t* v1, int64_t n, int passes,
                        const RadixScratch& R, const uint32_t* n_dev, const long long* max_dev, int* status,
                        cudaStream_t st) {
    constexpr int kTile = kSortBlock * kItems;
    const int64_t ntiles = (n + kTile - 1) / kTile;
    const int smem = (int)(sizeof(K) + (kVals ? 4 : 0)) * kTile;
    S* words = reinterpret_cast<S*>(R.words);
    for (int p = 0; p < passes; p++) {
        auto kern = kVals && p == 0 ? radix_pass_kernel<K, S, kVals, true, kItems>
                                       : radix_pass_kernel<K, S, kVals, false, kItems>;
        TDT_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        const K* kin = p == 0 ? in : (p & 1) ? b0 : b1;
        const uint32_t* vin = (p & 1) ? v0 : v1;
        kern<<<(unsigned)ntiles, kSortBlock, smem, st>>>(kin, vin, (p & 1) ? b1 : b0, (p & 1) ? v1 : v0, n, p,
                                                        R.hist + p * kRadix, R.tile_next + p,
                                                        words + (size_t)p * ntiles * kRadix, n_dev, max_dev,
                                                        look_back(status));
        TDT_LAUNCH_CHECK("radix_pass");
    }
    return TDT_OK;
}

template <class K, bool kVals>
int radix_sort(const K* in, K* b0, K* b1, uint32_t* v0, uint32_t* v1, int64_t n, int passes, const RadixScratch& R,
               const uint32_t* n_dev, const long long* max_dev, int* status, cudaStream_t st) {
    if (n <= 0) return TDT_OK;
    TDT_CHECK_ARG(n < (int64_t)UINT32_MAX, "radix sort of %lld keys exceeds 32-bit ranks", (long long)n);
    TDT_CHECK_ARG(passes >= 1 && passes <= kMaxPasses, "%d radix passes", passes);
    auto run = n < kSortSmall  ? radix_passes<K, uint32_t, kVals, kSortSmallItems>
               : n < kWideKeys ? radix_passes<K, uint32_t, kVals, kSortItems>
                               : radix_passes<K, unsigned long long, kVals, kSortItems>;
    return run(in, b0, b1, v0, v1, n, passes, R, n_dev, max_dev, status, st);
}

template int radix_sort<uint32_t, true>(const uint32_t*, uint32_t*, uint32_t*, uint32_t*, uint32_t*, int64_t, int,
                                        const RadixScratch&, const uint32_t*, const long long*, int*, cudaStream_t);
template int radix_sort<uint64_t, false>(const uint64_t*, uint64_t*, uint64_t*, uint32_t*, uint32_t*, int64_t, int,
                                         const RadixScratch&, const uint32_t*, const long long*, int*, cudaStream_t);

}  // namespace tdt
