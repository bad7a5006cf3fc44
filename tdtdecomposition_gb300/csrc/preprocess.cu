// Graph preprocessing on the device: raw edge list -> degree-oriented CSRCOO.
//
// Restates read_prepro_save (singlegpu_truss.py:172-178):
//   Graph.read_edgelist (src/type/Graph_Truss.py:177-213): drop self-loops
//     (:188), dedup unordered pairs (:200-202), rank vertices by degree
//     (:209-211; the reference's numpy argsort is unstable, here ties go to
//     the smaller id, and an optional vertex group ranks first so a batch of
//     graphs keeps contiguous rank ranges);
//   CSRCOO.edge_list_to_Graph (src/type/CSRCOO.py:128-162) + counter_sort
//     (:169-177): relabel by rank, orient low->high, CSR sorted by (row, col).
//
// Pipeline (every size that varies is read on the device, so there is no
// host synchronisation between the steps):
//   1. key = (min << B) | max per draw (self-loops -> sentinel), radix sort
//   2. keep the first of each run of equal keys (one pass with look-back) ->
//      E_out, and the degrees
//   3. present vertices -> (group, degree, id) keys, radix sort -> rank of
//      every id, vertices[rank]
//   4. relabel + orient each edge -> (lo << B) | hi, radix sort
//   5. rows / cols, and row_ptr from the places where the row changes
// Ids that come out of a sort are bounded before they index: a sort whose wait
// ran out leaves keys that are none (sort.cuh).
// Each sort's digit totals are taken by the kernel that makes its keys.  67 M /
// 65,536 draws: 10.6 ms / 560 us in 108 / 73 launches with five launches a sort
// pass and an atomic per degree and row count, 6.3 ms / 246 us in 26 / 18.
#include "common.cuh"
#include "sort.cuh"

namespace tdt {

static int bits_for(uint64_t x) {  // bits needed to hold values < x (x >= 1)
    int b = 0;
    while (b < 64 && (x - 1) >> b) b++;
    return b < 1 ? 1 : b;
}

constexpr int kPpBlock = 256;

__global__ void __launch_bounds__(kPpBlock) pp_edge_keys(const int32_t* __restrict__ src,
                                                         const int32_t* __restrict__ dst, int64_t m, int64_t num_ids,
                                                         int B, uint64_t sentinel, uint64_t* __restrict__ keys,
                                                         int passes, uint32_t* hist, int* status) {
    __shared__ uint32_t s_hist[kMaxPasses * kRadix];
    DigitHist H{s_hist};
    H.init(passes);
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < m; i += (int64_t)gridDim.x * blockDim.x) {
        const int32_t a = src[i], b = dst[i];
        uint64_t k = sentinel;
        if (a < 0 || b < 0 || a >= num_ids || b >= num_ids) {
            atomicMax(status, (int)TDT_ERR_INVALID);
        } else if (a != b) {
            const uint64_t lo = (uint64_t)(a < b ? a : b), hi = (uint64_t)(a < b ? b : a);
            k = (lo << B) | hi;
        }
        keys[i] = k;
        H.add(k, passes);
    }
    H.flush(passes, hist);
}

// Unique edges of the sorted keys (sentinels excluded), their number, and the
// degrees.  A tile's place comes from a look-back over the tiles before it.
// The sorted order gives a run of equal smaller ids one atomic per warp; the
// larger ids are random, and a hub among them would take its atomics one after
// the other, so a block counts the ids that come first to a slot of a small
// table in shared memory and adds those once, at its end.
constexpr int kUqItems = 8;
constexpr int kUqTile = kPpBlock * kUqItems;
constexpr int kUqTable = 2048;

struct UniqueCtl {
    unsigned long long next;
    uint32_t e_out;
};

__global__ void __launch_bounds__(kPpBlock) pp_unique(const uint64_t* __restrict__ keys, int64_t m,
                                                      uint64_t sentinel, int B, uint32_t num_ids,
                                                      uint64_t* __restrict__ ukeys,
                                                      int32_t* __restrict__ deg, unsigned long long* words,
                                                      UniqueCtl* ctl, LookBack L) {
    using W = TileWord<unsigned long long>;
    __shared__ int32_t s_id[kUqTable];
    __shared__ int32_t s_n[kUqTable];
    __shared__ uint32_t s_warp[kPpBlock / kWarp];
    __shared__ unsigned long long s_tile, s_before;
    const unsigned lane = lane_id();
    const unsigned lt = lanemask_lt();
    const int w = threadIdx.x / kWarp;
    const uint64_t mask = (1ull << B) - 1;
    const int64_t ntiles = (m + kUqTile - 1) / kUqTile;
    for (int i = threadIdx.x; i < kUqTable; i += kPpBlock) {
        s_id[i] = -1;
        s_n[i] = 0;
    }
    for (;;) {
        if (threadIdx.x == 0) s_tile = atomicAdd(&ctl->next, 1ull);
        __syncthreads();
        const int64_t tile = (int64_t)s_tile;
        if (tile >= ntiles) break;
        const int64_t base = tile * kUqTile + (int64_t)w * (kUqItems * kWarp);
        uint64_t k[kUqItems];
        unsigned f[kUqItems];
        uint32_t n = 0;
#pragma unroll
        for (int it = 0; it < kUqItems; it++) {
            const int64_t i = base + it * kWarp + lane;
            k[it] = i < m ? keys[i] : sentinel;
        }
        uint64_t last = base > 0 && base <= m ? keys[base - 1] : ~0ull;  // the key before this warp's
#pragma unroll
        for (int it = 0; it < kUqItems; it++) {
            uint64_t prev = __shfl_up_sync(kFull, k[it], 1);
            if (lane == 0) prev = last;
            last = __shfl_sync(kFull, k[it], 31);
            const bool first = base + it * kWarp + lane == 0 || k[it] != prev;
            f[it] = __ballot_sync(kFull, k[it] != sentinel && first);
            n += __popc(f[it]);
        }
        if (lane == 0) s_warp[w] = n;
        __syncthreads();
        uint32_t at = 0, tot = 0;
#pragma unroll
        for (int x = 0; x < kPpBlock / kWarp; x++) {
            const uint32_t c = s_warp[x];
            if (x < w) at += c;
            tot += c;
        }
        if (w == 0) {
            if (lane == 0) *(volatile unsigned long long*)(words + tile) = (tile == 0 ? W::kInclusive : W::kAggregate) | tot;
            const unsigned long long before = warp_look_back(words, tile, L);
            if (lane == 0) {
                if (tile > 0) *(volatile unsigned long long*)(words + tile) = W::kInclusive | (before + tot);
                s_before = before;
                if (tile == ntiles - 1) ctl->e_out = (uint32_t)(before + tot);
            }
        }
        // degrees, while the look-back runs
#pragma unroll
        for (int it = 0; it < kUqItems; it++) {
            if (f[it] == 0) continue;
            const bool mine = (f[it] >> lane) & 1u;
            const int32_t lo = (int32_t)(k[it] >> B), hi = (int32_t)(k[it] & mask);
            // runs of equal smaller ids among the lanes
            const int32_t plo = __shfl_up_sync(kFull, lo, 1);
            const unsigned heads = __ballot_sync(kFull, lane == 0 || plo != lo);
            const unsigned after = heads & ~(lt | (1u << lane));
            const unsigned run = ((after & (0u - after)) - 1u) & ~lt;  // from a head to before the next
            if ((heads >> lane) & 1u) {
                const int c = __popc(f[it] & run);
                if (c && (uint32_t)lo < num_ids) atomicAdd(deg + lo, c);
            }
            if (mine && (uint32_t)hi < num_ids) {
                const unsigned h = ((unsigned)hi * 2654435761u) >> 21;
                int32_t id = *(volatile int32_t*)(s_id + h);
                if (id == -1) id = atomicCAS(s_id + h, -1, hi);
                if (id == -1 || id == hi) atomicAdd(s_n + h, 1);
                else atomicAdd(deg + hi, 1);
            }
        }
        __syncthreads();
        int64_t to = (int64_t)s_before + at;
#pragma unroll
        for (int it = 0; it < kUqItems; it++) {
            if ((f[it] >> lane) & 1u) ukeys[to + __popc(f[it] & lt)] = k[it];
            to += __popc(f[it]);
        }
    }
    for (int i = threadIdx.x; i < kUqTable; i += kPpBlock)
        if (s_n[i]) atomicAdd(deg + s_id[i], s_n[i]);
}
static_assert(kUqTable == 1 << (32 - 21), "table index from the top bits of the product");

// vertex keys: present ids -> (group, degree, id); absent ids -> sentinel
__global__ void __launch_bounds__(kPpBlock) pp_vertex_keys(const int32_t* __restrict__ deg,
                                                           const int32_t* __restrict__ group, int64_t num_ids, int B,
                                                           int D, uint64_t* __restrict__ vkeys, int passes,
                                                           uint32_t* hist) {
    __shared__ uint32_t s_hist[kMaxPasses * kRadix];
    DigitHist H{s_hist};
    H.init(passes);
    for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < num_ids;
         v += (int64_t)gridDim.x * blockDim.x) {
        const int32_t d = deg[v];
        uint64_t k = ~0ull;
        if (d != 0) {
            const uint64_t g = group ? (uint64_t)group[v] : 0ull;
            k = (g << (B + D)) | ((uint64_t)d << B) | (uint64_t)v;
        }
        vkeys[v] = k;
        H.add(k, passes);
    }
    H.flush(passes, hist);
}

// sorted vertex keys -> rank[id], vertices[rank]; V_out = number of present ids
__global__ void pp_ranks(const uint64_t* __restrict__ vkeys, int64_t num_ids, int B, int32_t* __restrict__ rank,
                         int32_t* __restrict__ vertices, unsigned long long* __restrict__ vcount) {
    const uint64_t mask = (1ull << B) - 1;
    for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < num_ids;
         p += (int64_t)gridDim.x * blockDim.x) {
        const uint64_t k = vkeys[p];
        if (k == ~0ull) continue;
        const int32_t id = (int32_t)(k & mask);
        if (id >= num_ids) continue;
        rank[id] = (int32_t)p;
        vertices[p] = id;
        if (p + 1 == num_ids || vkeys[p + 1] == ~0ull) *vcount = (unsigned long long)(p + 1);
    }
}

// relabel the unique edges (last: the largest id)
__global__ void __launch_bounds__(kPpBlock) pp_relabel(const uint64_t* __restrict__ ukeys,
                                                       const uint32_t* __restrict__ e_out, int B,
                                                       const int32_t* __restrict__ rank,
                                                       uint64_t* __restrict__ keys2, uint32_t last, int passes,
                                                       uint32_t* hist) {
    __shared__ uint32_t s_hist[kMaxPasses * kRadix];
    DigitHist H{s_hist};
    H.init(passes);
    const uint64_t mask = (1ull << B) - 1;
    const int64_t eo = (int64_t)*e_out;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < eo; i += (int64_t)gridDim.x * blockDim.x) {
        const uint64_t k = ukeys[i];
        const uint64_t a = (uint64_t)rank[min((uint32_t)(k >> B), last)], b = (uint64_t)rank[min((uint32_t)(k & mask), last)];
        const uint64_t k2 = ((a < b ? a : b) << B) | (a < b ? b : a);
        keys2[i] = k2;
        H.add(k2, passes);
    }
    H.flush(passes, hist);
}

// rows, cols, and row_ptr: the rows after the one before an edge's, up to its
// own, start at the edge.  A lane fills short gaps itself, the warp long ones.
__global__ void pp_emit(const uint64_t* __restrict__ keys2, const uint32_t* __restrict__ e_out, int64_t num_ids,
                        int B, int32_t* __restrict__ rows, int32_t* __restrict__ cols,
                        int64_t* __restrict__ row_ptr) {
    const uint64_t mask = (1ull << B) - 1;
    const int64_t eo = (int64_t)*e_out;
    const unsigned lane = lane_id();
    const int64_t nth = (int64_t)gridDim.x * blockDim.x, tid = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    for (int64_t b = tid - lane; b < eo; b += nth) {
        const int64_t i = b + lane;
        int64_t r0 = 0, r1 = 0;  // rows [r0, r1) start at edge i
        if (i < eo) {
            const uint64_t k = keys2[i];
            const int32_t r = (int32_t)(k >> B);
            rows[i] = r;
            cols[i] = (int32_t)(k & mask);
            r1 = (int64_t)r + 1;
            r0 = i == 0 ? 0 : (int64_t)(keys2[i - 1] >> B) + 1;
            if (r < 0 || r >= num_ids) r0 = r1;
        }
        if (r1 - r0 <= 8)
            for (int64_t r = r0; r < r1; r++) row_ptr[r] = i;
        unsigned m = __ballot_sync(kFull, r1 - r0 > 8);
        while (m) {
            const int x = __ffs(m) - 1;
            m &= m - 1;
            const int64_t a = __shfl_sync(kFull, r0, x), c = __shfl_sync(kFull, r1, x);
            for (int64_t r = a + lane; r < c; r += kWarp) row_ptr[r] = b + x;
        }
    }
    // the rows after the last edge's, and the end
    const int64_t tail = eo > 0 ? (int64_t)(keys2[eo - 1] >> B) + 1 : 0;
    for (int64_t r = tail + tid; r <= num_ids; r += nth) row_ptr[r] = eo;
}

__global__ void pp_counts(const uint32_t* __restrict__ e_out, const unsigned long long* __restrict__ vcount,
                          const int* __restrict__ status, int64_t* __restrict__ counts) {
    counts[0] = (int64_t)*e_out;
    counts[1] = (int64_t)*vcount;
    counts[2] = *status;
}

namespace {
// Passes of the three sorts.
struct PpBits {
    int B, D, GB;
    int passes_e() const { return (2 * B + 7) / 8; }
    int passes_v() const { return (GB + D + B + 1 + 7) / 8; }
};

PpBits pp_bits(int64_t n, int32_t num_groups, bool grouped) {
    PpBits b;
    b.B = bits_for((uint64_t)n);
    b.D = bits_for((uint64_t)n + 1);  // degrees < num_ids in a simple graph
    b.GB = grouped ? bits_for((uint64_t)(num_groups > 0 ? num_groups : 1)) : 0;
    return b;
}

struct PpLayout {
    uint64_t* k0;
    uint64_t* k1;
    int32_t* rank;
    uint64_t* v0;
    uint64_t* v1;
    // zeroed in one go: counters, degrees, the unique pass's words, the sorts
    char* zero;
    size_t zero_bytes;
    int* status;
    unsigned long long* vcount;
    UniqueCtl* uniq;
    int32_t* deg;
    unsigned long long* uwords;
    RadixScratch se, sv, s2;
    size_t total;
};

PpLayout pp_carve(void* ws, int64_t m, int64_t n, int passes_e, int passes_v) {
    char* base = reinterpret_cast<char*>(ws);
    size_t off = 0;
    auto take = [&](size_t bytes) -> void* {
        off = (off + 255) & ~(size_t)255;
        void* p = base ? base + off : nullptr;
        off += bytes;
        return p;
    };
    const size_t M = (size_t)(m > 0 ? m : 1), N = (size_t)(n > 0 ? n : 1);
    PpLayout L;
    L.k0 = (uint64_t*)take(8 * M);
    L.k1 = (uint64_t*)take(8 * M);
    L.rank = (int32_t*)take(4 * N);
    L.v0 = (uint64_t*)take(8 * N);
    L.v1 = (uint64_t*)take(8 * N);
    char* misc = (char*)take(256);
    const size_t z0 = off - 256;
    L.zero = misc;
    L.status = (int*)misc;
    L.vcount = (unsigned long long*)(misc + 64);
    L.uniq = (UniqueCtl*)(misc + 128);
    L.deg = (int32_t*)take(4 * N);
    L.uwords = (unsigned long long*)take(8 * ((M + kUqTile - 1) / kUqTile));
    auto sort = [&](int64_t k, int passes) {
        const RadixScratch R = radix_scratch(nullptr, k, passes);
        return radix_scratch(take(R.bytes), k, passes);
    };
    L.se = sort((int64_t)M, passes_e);
    L.sv = sort((int64_t)N, passes_v);
    L.s2 = sort((int64_t)M, passes_e);
    L.zero_bytes = off - z0;
    L.total = off + 256;
    return L;
}
}  // namespace

// The workspace query does not know the groups: room for as many passes as
// keys can have.
size_t preprocess_workspace_bytes(int64_t m, int64_t n) {
    return pp_carve(nullptr, m, n, pp_bits(n > 0 ? n : 1, 0, false).passes_e(), kMaxPasses).total;
}

int run_preprocess(const int32_t* src, const int32_t* dst, int64_t m, int64_t num_ids, const int32_t* group,
                   int32_t num_groups, int32_t* rows, int32_t* cols, int64_t* row_ptr, int32_t* vertices,
                   int64_t* counts, void* ws, size_t ws_bytes, cudaStream_t st) {
    TDT_CHECK_ARG(m >= 0 && num_ids >= 0, "negative size");
    TDT_CHECK_ARG(m < (int64_t)UINT32_MAX - 1, "too many edges for one preprocessing call");
    TDT_CHECK_ARG(num_ids < (int64_t)INT32_MAX, "vertex ids must fit int32");
    TDT_CHECK_ARG(counts && row_ptr, "null output");
    TDT_CHECK_ARG(m == 0 || (src && dst && rows && cols), "null edge pointer");
    TDT_CHECK_ARG(num_ids == 0 || vertices, "null vertices");
    const size_t need = preprocess_workspace_bytes(m, num_ids);
    if (!ws || ws_bytes < need) {
        set_error("preprocess workspace of %zu bytes < required %zu", ws_bytes, need);
        return TDT_ERR_WORKSPACE;
    }
    DeviceInfo di;
    int rc = device_info(&di);
    if (rc) return rc;
    if (m == 0 || num_ids == 0) {
        TDT_CUDA(cudaMemsetAsync(row_ptr, 0, 8 * (size_t)(num_ids + 1), st));
        TDT_CUDA(cudaMemsetAsync(counts, 0, 3 * sizeof(int64_t), st));
        return TDT_OK;
    }
    const PpBits bits = pp_bits(num_ids, num_groups, group != nullptr);
    const int B = bits.B, D = bits.D;
    TDT_CHECK_ARG(2 * B + 1 <= 64 && B + D + bits.GB + 1 <= 64, "id/degree/group bits (%d/%d/%d) exceed 64", B, D,
                  bits.GB);
    const int pe = bits.passes_e(), pv = bits.passes_v();
    const PpLayout L = pp_carve(ws, m, num_ids, pe, pv);
    TDT_CUDA(cudaMemsetAsync(L.zero, 0, L.zero_bytes, st));
    const uint64_t sentinel = (1ull << (2 * B)) - 1;
    const int tb = kPpBlock;
    const unsigned g_m = grid_for(m, tb * 4, di.sms, 8), g_n = grid_for(num_ids, tb * 4, di.sms, 8);
    auto sorted = [](uint64_t* b0, uint64_t* b1, int passes) { return (passes & 1) ? b0 : b1; };
    // 1. edge keys, sorted (from k0 into k1 and back)
    pp_edge_keys<<<g_m, tb, 0, st>>>(src, dst, m, num_ids, B, sentinel, L.k0, pe, L.se.hist, L.status);
    TDT_LAUNCH_CHECK("pp_edge_keys");
    rc = radix_sort<uint64_t, false>(L.k0, L.k1, L.k0, nullptr, nullptr, m, pe, L.se, nullptr, nullptr, L.status, st);
    if (rc) return rc;
    uint64_t* sk = sorted(L.k1, L.k0, pe);
    uint64_t* uk = sk == L.k0 ? L.k1 : L.k0;
    // 2. dedup, degrees
    int per_sm = 0;
    TDT_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, pp_unique, kPpBlock, 0));
    pp_unique<<<grid_for(m, kUqTile, di.sms, per_sm > 0 ? per_sm : 1), kPpBlock, 0, st>>>(
        sk, m, sentinel, B, (uint32_t)num_ids, uk, L.deg, L.uwords, L.uniq, look_back(L.status));
    TDT_LAUNCH_CHECK("pp_unique");
    const uint32_t* e_out = &L.uniq->e_out;
    // 3. rank vertices by (group, degree, id); absent ids carry ~0, which stays
    // above every key on the low GB+D+B+1 bits
    pp_vertex_keys<<<g_n, tb, 0, st>>>(L.deg, group, num_ids, B, D, L.v0, pv, L.sv.hist);
    TDT_LAUNCH_CHECK("pp_vertex_keys");
    rc = radix_sort<uint64_t, false>(L.v0, L.v1, L.v0, nullptr, nullptr, num_ids, pv, L.sv, nullptr, nullptr, L.status,
                                     st);
    if (rc) return rc;
    pp_ranks<<<grid_for(num_ids, tb, di.sms, 16), tb, 0, st>>>(sorted(L.v1, L.v0, pv), num_ids, B, L.rank, vertices,
                                                              L.vcount);
    TDT_LAUNCH_CHECK("pp_ranks");
    // 4. relabel + orient, sort by (row, col); the sorted draw keys are no longer needed
    pp_relabel<<<g_m, tb, 0, st>>>(uk, e_out, B, L.rank, sk, (uint32_t)(num_ids - 1), pe, L.s2.hist);
    TDT_LAUNCH_CHECK("pp_relabel");
    rc = radix_sort<uint64_t, false>(sk, uk, sk, nullptr, nullptr, m, pe, L.s2, e_out, nullptr, L.status, st);
    if (rc) return rc;
    // 5. CSRCOO
    pp_emit<<<grid_for(m > num_ids ? m : num_ids, tb, di.sms, 16), tb, 0, st>>>(sorted(uk, sk, pe), e_out, num_ids, B,
                                                                               rows, cols, row_ptr);
    TDT_LAUNCH_CHECK("pp_emit");
    pp_counts<<<1, 1, 0, st>>>(e_out, L.vcount, L.status, counts);
    TDT_LAUNCH_CHECK("pp_counts");
    return TDT_OK;
}

}  // namespace tdt

extern "C" __attribute__((visibility("default"))) size_t tdt_preprocess_workspace_bytes(int64_t num_draws,
                                                                                       int64_t num_ids) {
    return tdt::preprocess_workspace_bytes(num_draws, num_ids);
}

extern "C" __attribute__((visibility("default"))) int tdt_preprocess(
    const int32_t* src, const int32_t* dst, int64_t num_draws, int64_t num_ids, const int32_t* vertex_group,
    int32_t num_groups, int32_t* rows, int32_t* cols, int64_t* row_ptr, int32_t* vertices, int64_t* counts,
    void* workspace, size_t workspace_bytes, tdt_stream_t stream) {
    return tdt::run_preprocess(src, dst, num_draws, num_ids, vertex_group, num_groups, rows, cols, row_ptr, vertices,
                               counts, workspace, workspace_bytes, (cudaStream_t)stream);
}
