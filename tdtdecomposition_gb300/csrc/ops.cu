// Drop-in `trusstensor` operators (myhpu_extension.cpp:572-593) for sm_103a.
//
// The reference runs one thread per (edge, tile) and walks a two-pointer merge
// of the two out-lists with scalar loads (kernel.cu:28-685).  Here a warp takes
// a group of edges and streams their N+(v) through a shared-memory table of
// N+(u) (walk_edges).  Matching on column values instead of merging keeps the
// operators exact on lists that carry the reference's -1 sentinels (peeled
// edges are overwritten with -1 in place, singlegpu_truss.py:118), where a
// binary search would not be.
//
// Tiling (n_cut): tile j of vertex v is [row_ptr[v*n_cut+j], row_ptr[v*n_cut+j+1])
// and tiles partition a row by column value (csr_to_tilingcsr,
// singlegpu_truss.py:160-169), so the union over tiles of the per-tile
// intersections is the intersection of the whole rows
// [row_ptr[v*n_cut], row_ptr[v*n_cut+n_cut]).
#include "common.cuh"

namespace tdt {

constexpr int kOpsBlock = 256;    // 8 warps
constexpr int kOpsMinBlocks = 5;  // resident blocks of the edge walks (shared memory)
constexpr int32_t kEmpty = INT32_MIN;

// Row ranges are clamped to [0, n_edges] so a malformed row_ptr cannot move an
// access outside the per-edge arrays.
struct RowView {
    const int32_t* rp;
    int32_t n_cut;
    int64_t nrows;    // vertices = (row_ptr_len - 1) / n_cut
    int64_t n_edges;
    __device__ __forceinline__ bool valid(int32_t v) const { return v >= 0 && v < nrows; }
    __device__ __forceinline__ int64_t clamp(int64_t x) const { return x < 0 ? 0 : (x > n_edges ? n_edges : x); }
    __device__ __forceinline__ int64_t begin(int32_t v) const { return clamp(__ldg(rp + (int64_t)v * n_cut)); }
    __device__ __forceinline__ int64_t end(int32_t v) const {
        int64_t b = begin(v), e = clamp(__ldg(rp + (int64_t)v * n_cut + n_cut));
        return e < b ? b : e;
    }
};

// ------------------------------------------------------------------ triangles of a list of edges
// For every edge (u, v) of a list, the columns that N+(u) and N+(v) share: the
// walk of the peel-update and k-truss operators.  A warp takes a group of list
// entries.  Edges of a group with the same u (neighbours in the list, as edges
// are stored by source) share one hash table of N+(u) in shared memory, with a
// bitmap of eight bits per slot in front of it; the rows N+(v) of these edges,
// widened to the aligned 16-byte chunks that hold them, form one flat space of
// chunks, walked 32 a step (the owner of a lane's chunk comes from one
// OR-reduction of the row starts inside the step).  A chunk that holds an entry
// is mapped as a whole, so any alignment of cols will do.  Most entries miss the
// bitmap; the others go to a queue and are looked up 32 at a time.  Rows of more
// than kWalkKeys keys are staged in pieces, or, where they are far longer than the
// run's N+(v) together, streamed (walk_long_run).
//
// Bound by issuing the tests.  One edge at a time, its shorter list hashed and
// the longer one streamed, the update of 0.87 M of 1.86 M edges (R-MAT scale 17,
// 109 M entries of N+(v)) took 540 us; in groups 416, with the counts of N+(u)
// kept in shared memory 431, in chunks of four columns 302 (2.4 M edges of a
// Chung-Lu graph 1,161 -> 564, the saturating support of all of scale 17
// 1,748 -> 770; without a case for wide rows in the loop 281).  Tables of 128 keys and more blocks per SM: 317.
constexpr int kWalkKeys = 256;                 // keys per pass, load factor <= 1/2
constexpr int kWalkSlots = 2 * kWalkKeys;
constexpr int kWalkMinLog2 = 6;
constexpr int kWalkQueue = 64;                 // a push adds up to 32 to at most 31
// Chunks of a run that is walked in groups: should all its entries be copies of one
// column, the count of their key fits 16 bits.
constexpr unsigned kWalkChunks = 65536 / 4 - 1;
constexpr int kLongRow = 512, kLongRatio = 2;

struct EdgeWalkShared {
    int32_t key[kWalkSlots];
    uint32_t bm[kWalkSlots / 4];
    uint4 row[kWarp];                          // N+(v) by place in the run: first chunk, begin, end, group lane
    uint2 queue[kWalkQueue];                   // ring: column, place in the run and offset in N+(v)
    uint32_t start[kWarp];                     // first chunk again
    int32_t cnt[kWarp];                        // by group lane
    uint32_t hits[kWalkKeys / 2];              // of each staged key, 16 bits
    uint16_t pos[kWalkSlots];                  // key index, and the flag of its edge in bit 15
};

// A table of up to kWalkKeys keys: log2 of its slots.
__device__ __forceinline__ int walk_table_log2(int d) {
    int lg = 33 - __clz(d);  // 2 d rounded up to a power of two, or the next one
    if (2 * d == 1 << (lg - 1)) lg--;
    return lg < kWalkMinLog2 ? kWalkMinLog2 : lg;
}

// A run whose N+(u) = [bu, eu) is long and kLongRatio times as long as its rows
// together (orders that are not degree ranks: a hub that ranks low), or one row
// past kWalkChunks: the keys of the rows are staged, piece by piece, each with its
// place in their flat space, and N+(u) is streamed.  Staged in pieces itself,
// such a row was streamed through once per 256 of its own keys.  Wheel of 200 K
// vertices, hub at id 0, update of 100 / 40,000 edges: 3.6 / 8.1 -> 1.1 / 2.5 ms
// (one edge at a time, the shorter row hashed: 1.5 / 4.5); 96 K vertices in
// cliques of 12 under such a hub 1.7 / 2.0 -> 0.53 / 0.78.  Longer rows or larger
// ratios as the line (1,024, 4,096; 8) measured the same.  In a turn of its own
// over the warp's groups: in the loop above it cost the update of R-MAT scale 17
// 1.8 %, as a call 10.
template <class Mark, class Hit, class Row>
__device__ __forceinline__ void walk_long_run(const int32_t* __restrict__ cols, EdgeWalkShared& S, unsigned run,
                                              int32_t bv, int32_t lv, unsigned marked, int64_t bu, int64_t eu,
                                              Mark&& mark, Hit&& hit, Row&& row) {
    const unsigned lane = lane_id(), lt = lanemask_lt();
    const unsigned shift = (unsigned)((uintptr_t)cols >> 2) & 3u;
    const int4* __restrict__ cols4 = reinterpret_cast<const int4*>(cols - shift);
    const bool mine = (run >> lane) & 1u;
    const unsigned incl = warp_incl_scan(mine ? (unsigned)lv : 0u);  // rows of different heads, or one: below 2^31
    const unsigned keys = __shfl_sync(kFull, incl, 31);
    const int places = __popc(run);
    if (mine) {  // by place in the run: keys before the row's, its first edge, its group lane
        const int k = __popc(run & lt);
        S.start[k] = incl - (unsigned)lv;
        S.row[k] = make_uint4(0u, (unsigned)bv, 0u, lane);
    }
    __syncwarp();
    auto place_of = [&](unsigned f) {
        int o = 0;
#pragma unroll
        for (int step = kWarp / 2; step > 0; step >>= 1)
            if (o + step < places && S.start[o + step] <= f) o += step;
        return o;
    };
    const unsigned ulo = (unsigned)bu + shift, uhi = (unsigned)eu + shift;
    const unsigned b0 = ulo >> 2, b1 = (uhi + 3) >> 2;
    for (unsigned c = 0; c < keys; c += kWalkKeys) {
        const int d = (int)(keys - c < kWalkKeys ? keys - c : kWalkKeys);
        const int lg = walk_table_log2(d);
        const unsigned slots = 1u << lg;
        for (unsigned k = lane; k < slots / 4; k += kWarp) {
            reinterpret_cast<int4*>(S.key)[k] = make_int4(kEmpty, kEmpty, kEmpty, kEmpty);
            S.bm[k] = 0u;
        }
        __syncwarp();
        for (int k = lane; k < d; k += kWarp) {
            const int o = place_of(c + k);
            const int32_t key = __ldg(cols + (int64_t)S.row[o].y + (c + k - S.start[o]));
            if (key < 0) continue;
            const unsigned h = (unsigned)key * 2654435761u;
            const unsigned bit = h >> (29 - lg);
            atomicOr(S.bm + (bit >> 5), 1u << (bit & 31));
            unsigned slot = h >> (32 - lg);
            while (atomicCAS(&S.key[slot], kEmpty, key) != kEmpty) slot = (slot + 1) & (slots - 1);
            S.pos[slot] = (uint16_t)k;
        }
        __syncwarp();
        int nq = 0;
        // look up the last m queue entries, one per lane: a key may be of several rows
        auto resolve = [&](int m) {
            __syncwarp();
            if ((int)lane < m) {
                const uint2 q = S.queue[nq - m + lane];
                const int64_t pb = (int64_t)q.y - shift;
                const bool mb = mark(pb);
                unsigned slot = (q.x * 2654435761u) >> (32 - lg);
                for (int32_t k = S.key[slot]; k != kEmpty; k = S.key[slot]) {
                    if (k == (int32_t)q.x) {
                        const unsigned f = c + S.pos[slot];
                        const int o = place_of(f);
                        const uint4 r = S.row[o];
                        const unsigned c2 = hit((marked >> r.w) & 1u, (int64_t)r.y + (f - S.start[o]), mb);
                        if (c2 & 1u) atomicAdd(&S.cnt[r.w], 1);
                        if (c2 & 2u) row(pb, 1);
                    }
                    slot = (slot + 1) & (slots - 1);
                }
            }
            __syncwarp();
            nq -= m;
        };
        for (unsigned b = b0; b < b1; b += kWarp) {
            const unsigned c4 = b + lane;
            unsigned cm = 0;
            int4 x4 = make_int4(0, 0, 0, 0);
            if (c4 < b1) {
                x4 = __ldg(cols4 + c4);
                auto test = [&](int32_t x) {
                    const unsigned t = ((unsigned)x * 2654435761u) >> (29 - lg);
                    return (S.bm[t >> 5] >> (t & 31)) & 1u;
                };
                cm = test(x4.x) | test(x4.y) << 1 | test(x4.z) << 2 | test(x4.w) << 3;
                if (4 * c4 < ulo) cm &= 0xFu << (ulo - 4 * c4);
                if (4 * c4 + 4 > uhi) cm &= 0xFu >> (4 * c4 + 4 - uhi);
            }
#pragma unroll 1
            for (int q = 0; q < 4; q++) {
                const int32_t x = q == 0 ? x4.x : q == 1 ? x4.y : q == 2 ? x4.z : x4.w;
                const bool cand = ((cm >> q) & 1u) && x >= 0;
                const unsigned m = __ballot_sync(kFull, cand);
                if (cand) S.queue[nq + __popc(m & lt)] = make_uint2((unsigned)x, 4 * c4 + (unsigned)q);
                nq += __popc(m);
                const bool end = q == 3 && b + kWarp >= b1;
                while (nq >= kWarp || (end && nq > 0)) resolve(nq < kWarp ? nq : kWarp);
            }
        }
    }
}

// list(i): the edge of entry i, or -1.  mark(e): flag of an edge.  hit(me, pa,
// mb): a common column, at position pa of N+(v) and an edge of u with flag mb;
// bit 0 of the result counts it for the entry's edge, bit 1 for the edge of u.
// row(pb, count) and done(e, count), count > 0: the counts of the edges of u, once
// per staged piece (of a long run hit by hit), and of the entries.  Long runs wait
// for a second turn over the warp's groups.
template <class List, class Mark, class Hit, class Row, class Done>
__device__ __forceinline__ void walk_edges(const int32_t* __restrict__ rows, const int32_t* __restrict__ cols,
                                           const RowView& rv, int64_t n, int group, EdgeWalkShared& S, List&& list,
                                           Mark&& mark, Hit&& hit, Row&& row, Done&& done) {
    const unsigned lane = lane_id(), lt = lanemask_lt();
    // chunk c of the flat space of positions + shift holds positions 4 c - shift .. + 3
    const unsigned shift = (unsigned)((uintptr_t)cols >> 2) & 3u;
    const int4* __restrict__ cols4 = reinterpret_cast<const int4*>(cols - shift);
    const int64_t nw = (int64_t)gridDim.x * (kOpsBlock / kWarp);
    const int64_t g0 = blockIdx.x * (int64_t)(kOpsBlock / kWarp) + threadIdx.x / kWarp;
    // a group's entries, one a lane (true: of a row that is to be walked)
    auto entry = [&](int64_t g, int64_t& e, int32_t& u, int32_t& bu, int32_t& eu, int32_t& bv, int32_t& lv, bool& me) {
        const int64_t i = g * group + lane;
        e = -1;
        u = -1;
        bu = eu = bv = lv = 0;
        me = false;
        if ((int)lane < group && i < n) {
            e = list(i);
            if (e >= 0 && e < rv.n_edges) {
                u = __ldg(rows + e);
                const int32_t v = __ldg(cols + e);
                if (rv.valid(u) && rv.valid(v)) {  // a sentinel edge has no triangles
                    bu = (int32_t)rv.begin(u);
                    eu = (int32_t)rv.end(u);
                    bv = (int32_t)rv.begin(v);
                    lv = (int32_t)(rv.end(v) - bv);
                    me = mark(e);
                }
            }
        }
        S.cnt[lane] = 0;
    };
    // the lanes of todo with the source of the first of them, and the chunks of
    // their rows: all of them, or the first where they are too many
    auto next_run = [&](unsigned todo, int first, int32_t u, int32_t bv, int32_t lv, bool wide, int32_t& start,
                        unsigned& total) {
        const int32_t ur = __shfl_sync(kFull, u, first);
        const unsigned lo = (unsigned)bv + shift, hi = lo + (unsigned)lv;
        const int32_t chunks = (int32_t)(((hi + 3) >> 2) - (lo >> 2));
        unsigned run = wide ? 1u << first : __ballot_sync(kFull, u == ur) & todo;
        const int32_t len = (run >> lane) & 1u ? chunks : 0;
        const int32_t incl = warp_incl_scan(len);
        start = incl - len;
        total = (unsigned)__shfl_sync(kFull, incl, 31);
        if (total > kWalkChunks && !wide) {
            run = 1u << first;
            start = 0;
            total = (unsigned)__shfl_sync(kFull, chunks, first);
        }
        return run;
    };
    auto is_long = [&](int64_t du, unsigned total) {
        return total > kWalkChunks || (du > kLongRow && du / (4 * kLongRatio) > (int64_t)total);
    };
    bool longs = false;
    for (int64_t g = g0; g * group < n; g += nw) {
        int64_t e;
        int32_t u, u0, u1, bv, lv;
        bool me;
        entry(g, e, u, u0, u1, bv, lv, me);
        const unsigned marked = __ballot_sync(kFull, me);
        const bool wide = __any_sync(kFull, lv >= (1 << 26));  // 32 of them might overflow a start
        unsigned todo = __ballot_sync(kFull, lv > 0);
        while (todo) {
            int32_t start;
            unsigned total;
            const int first = __ffs(todo) - 1;
            const unsigned run = next_run(todo, first, u, bv, lv, wide, start, total);
            todo &= ~run;
            const int64_t bu = __shfl_sync(kFull, u0, first), eu = __shfl_sync(kFull, u1, first);
            if (is_long(eu - bu, total)) {
                longs = true;
                continue;
            }
            if ((run >> lane) & 1u) {
                const int k = __popc(run & lt);
                const unsigned lo = (unsigned)bv + shift;
                S.start[k] = (unsigned)start;
                S.row[k] = make_uint4((unsigned)start, lo, lo + (unsigned)lv, lane);
            }
            const int nrun = __popc(run);
            for (int64_t c = bu; c < eu; c += kWalkKeys) {
                const int d = (int)(eu - c < kWalkKeys ? eu - c : kWalkKeys);
                const int lg = walk_table_log2(d);
                const unsigned slots = 1u << lg;
                for (unsigned k = lane; k < slots / 4; k += kWarp) {
                    reinterpret_cast<int4*>(S.key)[k] = make_int4(kEmpty, kEmpty, kEmpty, kEmpty);
                    S.bm[k] = 0u;
                }
                for (int k = lane; k < (d + 1) / 2; k += kWarp) S.hits[k] = 0u;
                __syncwarp();
                for (int k = lane; k < d; k += kWarp) {
                    const int32_t key = __ldg(cols + c + k);
                    if (key < 0) continue;
                    const unsigned h = (unsigned)key * 2654435761u;
                    const unsigned bit = h >> (29 - lg);
                    atomicOr(S.bm + (bit >> 5), 1u << (bit & 31));
                    unsigned slot = h >> (32 - lg);
                    while (atomicCAS(&S.key[slot], kEmpty, key) != kEmpty) slot = (slot + 1) & (slots - 1);
                    S.pos[slot] = (uint16_t)(k | (mark(c + k) ? 0x8000 : 0));
                }
                __syncwarp();
                int ob = 0, nq = 0;
                unsigned head = 0;
                // look up m queue entries, one per lane
                auto resolve = [&](int m) {
                    __syncwarp();
                    if ((int)lane < m) {
                        const uint2 q = S.queue[(head + lane) & (kWalkQueue - 1)];
                        const int32_t x = (int32_t)q.x;
                        const uint4 r = S.row[q.y & 31u];
                        unsigned slot = (q.x * 2654435761u) >> (32 - lg);
                        int32_t k = S.key[slot];
                        while (k != x && k != kEmpty) {
                            slot = (slot + 1) & (slots - 1);
                            k = S.key[slot];
                        }
                        if (k == x) {
                            const unsigned kb = S.pos[slot], at = kb & 0x7fffu;
                            const int64_t pa = (int64_t)r.y + (q.y >> 5) - shift;
                            const unsigned c2 = hit((marked >> r.w) & 1u, pa, (bool)(kb >> 15));
                            if (c2 & 1u) atomicAdd(&S.cnt[r.w], 1);
                            if (c2 & 2u) atomicAdd(&S.hits[at >> 1], 1u << (16 * (at & 1u)));
                        }
                    }
                    __syncwarp();
                    head += m;
                    nq -= m;
                };
                for (unsigned base = 0; base < total; base += kWarp) {
                    // row starts inside (base, base + 32): each is > base, and at most 31 fit
                    const int k = ob + 1 + (int)lane;
                    const unsigned B = k < nrun ? S.start[k] : ~0u;
                    const unsigned ahead = B - base;
                    const unsigned mk = __reduce_or_sync(kFull, ahead < (unsigned)kWarp ? 1u << ahead : 0u);
                    const int nb = __popc(mk);
                    const unsigned Bn = __shfl_sync(kFull, B, nb);
                    unsigned cm = 0, ent = 0;
                    int4 x4 = make_int4(0, 0, 0, 0);
                    if (base + lane < total) {
                        const int o = ob + __popc(mk & (lt | (1u << lane)));
                        const uint4 r = S.row[o];
                        const unsigned c4 = (r.y >> 2) + (base + lane - r.x), p0 = c4 << 2;
                        x4 = __ldg(cols4 + c4);
                        // every column is tested (a hashed index stays inside the
                        // bitmap); holes and entries outside the row are masked after
                        auto test = [&](int32_t x) {
                            const unsigned b = ((unsigned)x * 2654435761u) >> (29 - lg);
                            return (S.bm[b >> 5] >> (b & 31)) & 1u;
                        };
                        cm = test(x4.x) | test(x4.y) << 1 | test(x4.z) << 2 | test(x4.w) << 3;
                        if (p0 < r.y) cm &= 0xFu << (r.y - p0);
                        if (p0 + 4 > r.z) cm &= 0xFu >> (p0 + 4 - r.z);
                        ent = ((p0 - r.y) << 5) + (unsigned)o;
                    }
                    ob += nb + (Bn == base + kWarp ? 1 : 0);
                    const int32_t xs[4] = {x4.x, x4.y, x4.z, x4.w};
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        const bool cand = ((cm >> q) & 1u) && xs[q] >= 0;
                        const unsigned m = __ballot_sync(kFull, cand);
                        if (cand)
                            S.queue[(head + nq + __popc(m & lt)) & (kWalkQueue - 1)] =
                                make_uint2((unsigned)xs[q], ent + ((unsigned)q << 5));
                        nq += __popc(m);
                        if (nq >= kWarp) resolve(kWarp);
                    }
                }
                if (nq > 0) resolve(nq);
                __syncwarp();
                for (int k = lane; k < d; k += kWarp) {
                    const int32_t count = (int32_t)((S.hits[k >> 1] >> (16 * (k & 1))) & 0xffffu);
                    if (count > 0) row(c + k, count);
                }
                __syncwarp();
            }
        }
        const int32_t count = S.cnt[lane];
        if (count > 0) done(e, count);
        __syncwarp();
    }
    if (!longs) return;
    for (int64_t g = g0; g * group < n; g += nw) {
        int64_t e;
        int32_t u, u0, u1, bv, lv;
        bool me;
        entry(g, e, u, u0, u1, bv, lv, me);
        const unsigned marked = __ballot_sync(kFull, me);
        const bool wide = __any_sync(kFull, lv >= (1 << 26));
        unsigned todo = __ballot_sync(kFull, lv > 0);
        while (todo) {
            int32_t start;
            unsigned total;
            const int first = __ffs(todo) - 1;
            const unsigned run = next_run(todo, first, u, bv, lv, wide, start, total);
            todo &= ~run;
            const int64_t bu = __shfl_sync(kFull, u0, first), eu = __shfl_sync(kFull, u1, first);
            if (is_long(eu - bu, total)) walk_long_run(cols, S, run, bv, lv, marked, bu, eu, mark, hit, row);
            __syncwarp();
        }
        const int32_t count = S.cnt[lane];
        if (count > 0) done(e, count);
        __syncwarp();
    }
}

// Entries a warp takes at a time: as many as leave every warp of the grid
// kWalkTurns groups, at most a warp's width; 4 or 8 turns measured the same.
constexpr int kWalkTurns = 2;

// ------------------------------------------------------------------ segment_add
// kernel.cu:5-26: one thread per row.
__global__ void segment_add_kernel(const int32_t* __restrict__ vals, const int32_t* __restrict__ ptr,
                                   int32_t* __restrict__ out, int64_t nrows, int64_t nvals) {
    for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < nrows;
         r += (int64_t)gridDim.x * blockDim.x) {
        int32_t s = __ldg(ptr + r), e = __ldg(ptr + r + 1);
        if (nvals >= 0) {  // clamp to the values array when its length is known
            s = s < 0 ? 0 : (s > nvals ? (int32_t)nvals : s);
            e = e < 0 ? 0 : (e > nvals ? (int32_t)nvals : e);
        }
        if (s < e) {
            int32_t sum = 0;
            for (int32_t i = s; i < e; i++) sum += __ldg(vals + i);
            out[r] = sum;
        }
    }
}

// ------------------------------------------------------------------ segment_max
// out[g] = max(out[g], values of segment g): the per-graph kmax of a batch.
// One pass over the values.  Each warp owns one contiguous slab, finds the
// segment of its first value by binary search and walks on from there, so a
// long segment spreads over many warps and a slab of short ones stays in one;
// one atomic per (slab, segment).  Bound by reading the values; one 64-bit
// atomic per value on the segments' addresses (14 M values, 512 segments) took
// 5.6 ms of an 11.7 ms batch, which took 5.9 ms with this kernel (4.7 ms now).
constexpr int kSegMaxUnroll = 4;

__global__ void __launch_bounds__(kOpsBlock) segment_max_kernel(const int32_t* __restrict__ vals,
                                                                const int64_t* __restrict__ off, int64_t nseg,
                                                                int64_t nvals, int64_t slab,
                                                                long long* __restrict__ out) {
    const unsigned lane = lane_id();
    const int64_t w = (blockIdx.x * (int64_t)kOpsBlock + threadIdx.x) / kWarp;
    int64_t p = w * slab;
    const int64_t pe = p + slab < nvals ? p + slab : nvals;
    if (p >= pe) return;
    int64_t g = 0, hi = nseg;  // first segment that ends past p
    while (g < hi) {
        const int64_t mid = (g + hi) >> 1;
        if (__ldg(off + mid + 1) <= p) g = mid + 1; else hi = mid;
    }
    for (; g < nseg; g++) {
        const int64_t b = __ldg(off + g), e = __ldg(off + g + 1);
        if (b >= pe) break;
        p = p < b ? b : p;
        const int64_t end = e < pe ? e : pe;
        int32_t m = INT32_MIN;
        for (int64_t i = p + lane; i < end; i += kSegMaxUnroll * kWarp) {
            int32_t x[kSegMaxUnroll];
#pragma unroll
            for (int k = 0; k < kSegMaxUnroll; k++) x[k] = i + k * kWarp < end ? __ldg(vals + i + k * kWarp) : INT32_MIN;
#pragma unroll
            for (int k = 0; k < kSegMaxUnroll; k++) m = x[k] > m ? x[k] : m;
        }
        if (p < end) {
            m = __reduce_max_sync(kFull, m);
            if (lane == 0) atomicMax(out + g, (long long)m);
            p = end;
        }
    }
}

// ------------------------------------------------------------------ max_id
// Bound by its launch on small inputs and by the read on large ones: two
// reductions and a maximum of a general library took 38 us of a preprocessing
// of 65,536 draws.
__global__ void __launch_bounds__(kOpsBlock) max_id_kernel(const int32_t* __restrict__ a, int64_t na,
                                                           const int32_t* __restrict__ b, int64_t nb, int32_t* out) {
    constexpr int kUnroll = 8;
    const int64_t step = (int64_t)gridDim.x * kOpsBlock;
    int32_t m = INT32_MIN;
    auto scan = [&](const int32_t* __restrict__ x, int64_t n) {
        for (int64_t i = blockIdx.x * (int64_t)kOpsBlock + threadIdx.x; i < n; i += kUnroll * step) {
            int32_t v[kUnroll];
#pragma unroll
            for (int k = 0; k < kUnroll; k++) v[k] = i + k * step < n ? __ldg(x + i + k * step) : INT32_MIN;
#pragma unroll
            for (int k = 0; k < kUnroll; k++) m = v[k] > m ? v[k] : m;
        }
    };
    scan(a, na);
    scan(b, nb);
    m = __reduce_max_sync(kFull, m);
    if (lane_id() == 0 && m > *(volatile int32_t*)out) atomicMax(out, m);
}

// ------------------------------------------------------------------ peel-update operators
enum AffectMode { kAffectDeleted = 0, kAffectNot = 1, kAffectNotWin = 2 };

struct AffectArgs {
    const int32_t* e_affect;
    int64_t n_affect;
    const int32_t* rows;
    const int32_t* cols;
    RowView rv;
    const uint8_t* mark;
    int32_t l;
    uint8_t* n_mark;
    int32_t* out;
    int32_t windows_high;
    uint8_t* in_win;
    int32_t* buff_index;
    int32_t* buf_size;
    int group;
};

// kernel.cu:144-191/:407-456 (kAffectDeleted), :220-273/:492-547 (kAffectNot),
// :302-370/:578-648 (kAffectNotWin).
template <int MODE>
__global__ void __launch_bounds__(kOpsBlock, kOpsMinBlocks) affect_kernel(AffectArgs A) {
    __shared__ __align__(16) EdgeWalkShared s[kOpsBlock / kWarp];
    auto in_window = [&](int64_t x) {
        A.in_win[x] = 1;
        const int32_t slot = atomicAdd(A.buf_size, 1);
        if (slot >= 0 && slot < A.rv.n_edges) A.buff_index[slot] = (int32_t)x;
    };
    auto lower = [&](int64_t x, int32_t by) {
        const int32_t t = atomicSub(A.out + x, by);
        if (MODE == kAffectDeleted || (t > A.l && t - by <= A.l)) A.n_mark[x] = 1;
        if (MODE == kAffectNotWin && t >= A.windows_high && t - by < A.windows_high) in_window(x);
    };
    walk_edges(
        A.rows, A.cols, A.rv, A.n_affect, A.group, s[threadIdx.x / kWarp],
        [&](int64_t i) { return (int64_t)__ldg(A.e_affect + i); }, [&](int64_t e) { return A.mark[e] != 0; },
        [&](bool me, int64_t pa, bool mb) {
            const bool ma = A.mark[pa] != 0;
            const int32_t now = *(volatile int32_t*)(A.out + pa);
            if (MODE == kAffectDeleted ? !(me || ma || mb) : me && ma && mb) return 0u;
            if (now > A.l) lower(pa, 1);
            return (MODE == kAffectDeleted ? !me : me) ? 3u : 2u;
        },
        [&](int64_t pb, int32_t count) {
            // as far as one after the other would: a value falls while it is above l
            const int32_t now = *(volatile int32_t*)(A.out + pb);
            if (now > A.l) lower(pb, (int32_t)min((int64_t)count, (int64_t)now - A.l));
        },
        [&](int64_t e, int32_t count) {
            int32_t t = atomicSub(A.out + e, count);
            if (MODE == kAffectDeleted || t - count <= A.l) A.n_mark[e] = 1;
            if (MODE == kAffectNotWin && t - count < A.windows_high && t >= A.windows_high) in_window(e);
        });
}

// ------------------------------------------------------------------ k-truss search operators
struct EdgeOpArgs {
    const int32_t* rows;
    const int32_t* cols;
    RowView rv;
    int64_t n_edges;
    int32_t k;
    const uint8_t* mark;
    int32_t* out;
    int group;
};

// ktruss_cuda.py:121-200: support saturating at k.
__global__ void __launch_bounds__(kOpsBlock, kOpsMinBlocks) support_k_kernel(EdgeOpArgs A) {
    __shared__ __align__(16) EdgeWalkShared s[kOpsBlock / kWarp];
    walk_edges(
        A.rows, A.cols, A.rv, A.n_edges, A.group, s[threadIdx.x / kWarp], [](int64_t i) { return i; },
        [](int64_t) { return false; },
        [&](bool, int64_t pa, bool) {
            if (*(volatile int32_t*)(A.out + pa) < A.k) atomicAdd(A.out + pa, 1);
            return 3u;
        },
        [&](int64_t pb, int32_t count) {
            const int32_t now = *(volatile int32_t*)(A.out + pb);
            if (now < A.k) atomicAdd(A.out + pb, (int32_t)min((int64_t)count, (int64_t)A.k - now));
        },
        [&](int64_t e, int32_t count) {
            if (*(volatile int32_t*)(A.out + e) < A.k) atomicAdd(A.out + e, count);
        });
}

// ktruss_cuda.py:201-286: unconditional decrements on an extracted subgraph.
__global__ void __launch_bounds__(kOpsBlock, kOpsMinBlocks) sub_affect_kernel(EdgeOpArgs A) {
    __shared__ __align__(16) EdgeWalkShared s[kOpsBlock / kWarp];
    walk_edges(
        A.rows, A.cols, A.rv, A.n_edges, A.group, s[threadIdx.x / kWarp], [](int64_t i) { return i; },
        [&](int64_t e) { return A.mark[e] != 0; },
        [&](bool me, int64_t pa, bool mb) {
            const bool ma = A.mark[pa] != 0;
            if (!(me || ma || mb)) return 0u;
            if (!ma) atomicSub(A.out + pa, 1);
            return (me ? 0u : 1u) | (mb ? 0u : 2u);
        },
        [&](int64_t pb, int32_t count) { atomicSub(A.out + pb, count); },
        [&](int64_t e, int32_t count) { atomicSub(A.out + e, count); });
}

// ------------------------------------------------------------------ host launchers
// Grid of a walk over n list entries, and the entries a warp takes at a time.
static int walk_grid(int64_t n, int* group) {
    DeviceInfo di;
    if (device_info(&di) != TDT_OK) return -1;
    const int64_t warps = (int64_t)di.sms * kOpsMinBlocks * (kOpsBlock / kWarp);
    int64_t per = n / (warps * kWalkTurns);
    if (per < 1) per = 1;
    if (per > kWarp) per = kWarp;
    *group = (int)per;
    const int64_t groups = (n + per - 1) / per;
    const int64_t blocks = (groups + kOpsBlock / kWarp - 1) / (kOpsBlock / kWarp), cap = (int64_t)di.sms * kOpsMinBlocks;
    return (int)(blocks < cap ? blocks : cap);
}

static int check_rowptr(int64_t row_ptr_len, int32_t n_cut) {
    TDT_CHECK_ARG(n_cut >= 1, "n_cut must be >= 1 (got %d)", n_cut);
    TDT_CHECK_ARG(row_ptr_len >= 1 && (row_ptr_len - 1) % n_cut == 0,
                  "row_ptr length %lld is not V*n_cut+1 for n_cut=%d", (long long)row_ptr_len, n_cut);
    return TDT_OK;
}

int launch_segment_add(const int32_t* vals, const int32_t* ptr, int32_t* out, int64_t nrows, int64_t nvals,
                       cudaStream_t st) {
    TDT_CHECK_ARG(nrows >= 0, "num_rows < 0");
    if (nrows == 0) return TDT_OK;
    TDT_CHECK_ARG(vals && ptr && out, "null pointer");
    DeviceInfo di;
    int rc = device_info(&di);
    if (rc) return rc;
    segment_add_kernel<<<grid_for(nrows, 256, di.sms, 16), 256, 0, st>>>(vals, ptr, out, nrows, nvals);
    TDT_LAUNCH_CHECK("segment_add");
    return TDT_OK;
}

int launch_segment_max(const int32_t* vals, const int64_t* off, int64_t nseg, int64_t nvals, int64_t* out,
                       cudaStream_t st) {
    TDT_CHECK_ARG(nseg >= 0 && nvals >= 0, "negative size");
    if (nseg == 0 || nvals == 0) return TDT_OK;
    TDT_CHECK_ARG(vals && off && out, "null pointer");
    DeviceInfo di;
    int rc = device_info(&di);
    if (rc) return rc;
    // whole steps of a warp, at most one wave of 8 blocks per SM
    constexpr int64_t step = kSegMaxUnroll * kWarp;
    const int64_t warps = (int64_t)di.sms * 8 * (kOpsBlock / kWarp);
    int64_t slab = ((nvals + warps - 1) / warps + step - 1) / step * step;
    const int64_t used = (nvals + slab - 1) / slab;
    const unsigned blocks = (unsigned)((used + kOpsBlock / kWarp - 1) / (kOpsBlock / kWarp));
    segment_max_kernel<<<blocks, kOpsBlock, 0, st>>>(vals, off, nseg, nvals, slab,
                                                     reinterpret_cast<long long*>(out));
    TDT_LAUNCH_CHECK("segment_max");
    return TDT_OK;
}

int launch_max_id(const int32_t* a, int64_t na, const int32_t* b, int64_t nb, int32_t* out, cudaStream_t st) {
    TDT_CHECK_ARG(na >= 0 && nb >= 0, "negative size");
    TDT_CHECK_ARG(out && (a || na == 0) && (b || nb == 0), "null pointer");
    DeviceInfo di;
    int rc = device_info(&di);
    if (rc) return rc;
    TDT_CUDA(cudaMemsetAsync(out, 0x80, sizeof(int32_t), st));
    const int64_t n = na > nb ? na : nb;
    if (n == 0) return TDT_OK;
    max_id_kernel<<<grid_for(n, kOpsBlock, di.sms, 8), kOpsBlock, 0, st>>>(a, na, b, nb, out);
    TDT_LAUNCH_CHECK("max_id");
    return TDT_OK;
}

int launch_affect(int mode, const int32_t* e_affect, int64_t n_affect, const int32_t* rows,
                  const int32_t* cols, const int32_t* rp, int64_t row_ptr_len, int32_t n_cut,
                  const uint8_t* mark, int32_t l, uint8_t* n_mark, int32_t* out, int32_t windows_high,
                  uint8_t* in_win, int32_t* buff_index, int32_t* buf_size, int64_t n_edges,
                  cudaStream_t st) {
    int rc = check_rowptr(row_ptr_len, n_cut);
    if (rc) return rc;
    TDT_CHECK_ARG(n_affect >= 0 && n_edges >= 0, "negative size");
    if (n_affect == 0) return TDT_OK;
    TDT_CHECK_ARG(e_affect && rows && cols && rp && mark && n_mark && out, "null pointer");
    if (mode == kAffectNotWin) TDT_CHECK_ARG(in_win && buff_index && buf_size, "null window buffer");
    AffectArgs A{e_affect, n_affect, rows, cols, RowView{rp, n_cut, (row_ptr_len - 1) / n_cut, n_edges},
                 mark, l, n_mark, out, windows_high, in_win, buff_index, buf_size, 0};
    int g = walk_grid(n_affect, &A.group);
    if (g < 0) return TDT_ERR_CUDA;
    switch (mode) {
        case kAffectDeleted: affect_kernel<kAffectDeleted><<<g, kOpsBlock, 0, st>>>(A); break;
        case kAffectNot: affect_kernel<kAffectNot><<<g, kOpsBlock, 0, st>>>(A); break;
        default: affect_kernel<kAffectNotWin><<<g, kOpsBlock, 0, st>>>(A); break;
    }
    TDT_LAUNCH_CHECK("affect");
    return TDT_OK;
}

int launch_support_k(const int32_t* rows, const int32_t* cols, const int32_t* rp, int64_t row_ptr_len,
                     int32_t n_cut, int32_t k, int32_t* out, int64_t n_edges, cudaStream_t st) {
    int rc = check_rowptr(row_ptr_len, n_cut);
    if (rc) return rc;
    TDT_CHECK_ARG(n_edges >= 0, "negative size");
    if (n_edges == 0) return TDT_OK;
    TDT_CHECK_ARG(rows && cols && rp && out, "null pointer");
    EdgeOpArgs A{rows, cols, RowView{rp, n_cut, (row_ptr_len - 1) / n_cut, n_edges}, n_edges, k, nullptr, out, 0};
    int g = walk_grid(n_edges, &A.group);
    if (g < 0) return TDT_ERR_CUDA;
    support_k_kernel<<<g, kOpsBlock, 0, st>>>(A);
    TDT_LAUNCH_CHECK("support_k");
    return TDT_OK;
}

int launch_sub_affect(const int32_t* rows, const int32_t* cols, const int32_t* rp, int64_t row_ptr_len,
                      int32_t n_cut, const uint8_t* mark, int32_t* out, int64_t n_edges,
                      cudaStream_t st) {
    int rc = check_rowptr(row_ptr_len, n_cut);
    if (rc) return rc;
    TDT_CHECK_ARG(n_edges >= 0, "negative size");
    if (n_edges == 0) return TDT_OK;
    TDT_CHECK_ARG(rows && cols && rp && mark && out, "null pointer");
    EdgeOpArgs A{rows, cols, RowView{rp, n_cut, (row_ptr_len - 1) / n_cut, n_edges}, n_edges, 0, mark, out, 0};
    int g = walk_grid(n_edges, &A.group);
    if (g < 0) return TDT_ERR_CUDA;
    sub_affect_kernel<<<g, kOpsBlock, 0, st>>>(A);
    TDT_LAUNCH_CHECK("sub_affect");
    return TDT_OK;
}

}  // namespace tdt
