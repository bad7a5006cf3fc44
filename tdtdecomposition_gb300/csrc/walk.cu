// The triangle walk of the whole-path calls: per-edge role counts and per-edge
// triangle lists over the degree-oriented CSR.
//
// A triangle (u, v, w), u -> v, u -> w, v -> w, has the edges eA = (u,v)
// (source, middle), eB = (u,w) (source, sink) and eC = (v,w) (middle, sink).
// It is found from its MIDDLE vertex v: N+(v) is staged once and the tails
// N+(u)[i+1..) of the in-edges (u,v), v = N+(u)[i], are streamed through it.
// Walking from the source u instead streams all of N+(v) for every (u,v):
// the out-list of a high-ranked middle vertex is longer than the tail behind
// it, 660 M against 205 M entries at R-MAT scale 18 (83 M triangles), 257 M
// against 63 M on a Chung-Lu graph of 200 K vertices.
//
// * Row v (at most the buffer's entries; longer rows in column chunks) is a
//   bitmap over w - wb, sixteen bits a word with the running count of the
//   words before it in the upper half.  Ids are degree ranks, so N+(v) of the
//   vertices with most of the work lies in a narrow range: then the bitmap is
//   exact and one shared-memory load answers both whether w is in N+(v) and
//   where (prefix plus one popcount).  A wider row indexes by the low bits of
//   w - wb: the rank leads to an entry of the row that is compared with w, and
//   ids that share a bit are searched for.
// * Rows with next to no work are not staged: a warp takes the in-edges of up
//   to 32 of them together and searches each row in place.
// * A row with few in-edges belongs to one warp (2^13-bit bitmap); one with
//   many, or with more than warp_cap out-edges, to a block (2^16 bits) whose
//   warps take its in-edges 32 at a time.  The in-edges of a hub are split
//   into parts of kPart, each a unit of its own.
// * A tail far longer than the row is not streamed: the row's entries are
//   searched in it, at the end of the warp's work (walk_long_tails).
// * The tails of 32 in-edges form one flat space of 16-byte chunks of cols: a
//   lane loads four columns per step and the owning in-edge of each lane's
//   chunk comes from one OR-reduction over the group's starts.
// * The role-A entries (eB, eC) of an in-edge come out together and are stored
//   side by side (a warp owns the tail; positions from ballots).  Role C is
//   counted in shared memory with the row, role A with the group; only role B
//   takes a global reduction.
// * Roles B and C are the role-A entries regrouped by row and by middle vertex
//   (distribute_kernel): each chunk is sorted by target edge in shared memory
//   and written out in runs.  Scattered 8-byte stores reach 190 G/s into L2
//   and 22 G/s past it, runs of eight 640 and 115 G/s (measured).
//
// One walk counts and lists when the list tail has room for a staging region
// per edge as well: (u,v) at position i of a row of d holds at most d - i - 1
// role-A entries, so the regions of a row take d (d - 1) / 2 slots and every
// start is a formula over the rows' scanned totals.  Without that room the
// count walk is followed by a list walk.
//
// Measured at R-MAT scale 20 / 22 (support + listing, against a walk from the
// source with staged entries, compaction and transposition): 21.5 -> 13.7 ms,
// 106 -> 73.6 ms; the count alone, with its in-adjacency, at scale 21: 19.3 ->
// 7.7 ms.  The walk issues 2.6 instructions a cycle per SM (scale 20: 4.1 ms,
// DRAM 29 %); the regrouping moves 13 GB in 4 ms per role.
#include "common.cuh"
#include "sort.cuh"

namespace tdt {

constexpr int kWkBlock = 256;
constexpr int kWkWarps = kWkBlock / kWarp;
constexpr int kWkMinBlocks = 5;
// In-edges per unit of a block row, and past which a v is a hub: its windows of
// the role-C pass pay a global atomic per run (listing at R-MAT scale 22: 61 ms
// with 2,048, 49 with 4,096, 47 with 16,384), where a whole hub in one block
// is a long last window (Chung-Lu, 1 M vertices: 10.2 ms unsplit, 7.1 split).
constexpr int kPart = 16384;
// Rows with at most this many in-edges go to one warp.  Fewer block rows mean
// fewer barriers, more of them a shorter last warp: 32 against 128 measured
// 0.31 / 0.42 ms of support phase at R-MAT scale 16 (0.9 M edges), 1.38 / 1.29
// at 18 (3.8 M), 30.6 / 28.8 at 22 (64 M).
constexpr int kLightInSmall = 32, kLightInLarge = 128;
constexpr int64_t kLightInEdges = 1 << 21;
constexpr int kTopBatch = 2;         // light rows per grab in the top quarter of the ranks
constexpr int kLightCap = 256;       // and at most this many out-edges
constexpr int kLightLog2 = 13;
constexpr int kHeavyLog2 = 16;
constexpr int kRowCap = 4096;        // out-edges of a block row (or of one of its column chunks)
constexpr int kLightWords = (1 << kLightLog2) / 16;
constexpr int kHeavyWords = (1 << kHeavyLog2) / 16;

// Shared memory: the block row, aliased by the warps' light rows, then one
// group per warp (int4 GE[32], entry offsets int64[32], counters u32[32]).
constexpr int kWkBm = 0;
constexpr int kWkCnt = kWkBm + 4 * kHeavyWords;
constexpr int kWkRowBytes = kWkCnt + 4 * kRowCap;
constexpr int kLtBm = 0;
constexpr int kLtCnt = kLtBm + 4 * kLightWords;
constexpr int kLtPerm = kLtCnt + 4 * kLightCap;
constexpr int kLtBytes = kLtPerm + kLightCap;
static_assert(kLtBytes % 16 == 0 && kLtBytes * kWkWarps <= kWkRowBytes, "light rows alias the block row");
static_assert(kRowCap < 65536 && kLightCap <= 256, "16-bit prefixes, 8-bit entries of the light rows");
constexpr int kGrpBytes = kWarp * (16 + 8 + 4);
constexpr int kWkSmem = kWkRowBytes + kWkWarps * kGrpBytes;
static_assert(kWkRowBytes % 16 == 0 && kGrpBytes % 16 == 0, "group alignment");

enum WalkMode { kWalkCount = 0, kWalkList = 1 };

struct WalkArgs {
    const int64_t* rp;
    const int32_t* cols;
    const int64_t* cp;          // in-adjacency: offsets, source vertices, edge ids
    const int32_t* in_src;
    const int32_t* in_eid;
    int64_t nv, ne;
    int32_t* cA;                // role counts: written by kWalkCount (zeroed before), read by kWalkList
    int32_t* cB;
    int32_t* cC;
    const int64_t* sbase;       // kWalkCount: staging slots before each row, sbase[nv] in all (null: count only)
    const int64_t* off;         // kWalkList: list offsets int64[E+1]
    int2* out;                  // kWalkCount: end of the staging slots; kWalkList: the lists
    int32_t* runA;              // role-A entries so far of rows walked in column chunks
    uint32_t* longs;            // per in-edge with a long tail: the lane's one before it (walk_long_tails)
    const int2* units;          // block rows: {v, part}
    int* status;
    const int* gate;            // non-zero: skip
    const int* stage_skip;      // kWalkCount: non-zero: count only (written by the plan)
    int warp_cap;
    int light_in;
    int row_cap;
};

struct WalkCtl {
    unsigned long long nunits, nhubs; // written by the plan
    unsigned long long unit_next[2];  // work counters of the count and the list walk
    unsigned long long light_next[2];
    unsigned long long dist_next[2];  // and of the role-B and role-C passes
    unsigned long long dist_done;     // blocks that finished the role-C pass
};

// First staging slot of the role-A entries of the edge at position i of a row
// of d edges whose slots start at base.
__device__ __forceinline__ int64_t stage_slot(int64_t base, int64_t d, int64_t i) {
    return base + i * (2 * d - 1 - i) / 2;
}

// Test knobs shared with the drop-in support operator (support.cu).
void support_caps(int* warp_cap, int* heavy_cap);

// Rows searched in place instead of staged: din searches of log2(dout) steps
// cost less than clearing and filling a bitmap (support phase of 512
// Barabasi-Albert graphs 2.05 ms without, 1.86 with 64, 1.88 with 128).
constexpr int kTinySteps = 64;
__device__ __forceinline__ bool is_tiny_row(int dout, int din) { return din * (32 - __clz(dout)) <= kTinySteps; }

// The hubs follow the units in the plan's scratch.
static int32_t* hub_list(void* units, int64_t ne) { return reinterpret_cast<int32_t*>(reinterpret_cast<int2*>(units) + ne); }

__device__ __forceinline__ bool is_block_row(int64_t dout, int64_t din, int warp_cap, int light_in) {
    return dout > warp_cap || din > light_in;
}

// Units of the block rows, one per kPart in-edges (Sum of ceil(d- / kPart)
// over rows with in-edges is at most E), and the hubs, the rows of several.
__global__ void walk_plan_kernel(const int64_t* __restrict__ rp, const int64_t* __restrict__ cp, int64_t nv,
                                 int warp_cap, int light_in, int2* __restrict__ units,
                                 int32_t* __restrict__ hubs, const int64_t* __restrict__ sbase,
                                 unsigned long long stage_slots, int* stage_skip, WalkCtl* ctl, const int* status) {
    if (blockIdx.x == 0 && threadIdx.x == 0)
        *stage_skip = !(*(volatile const int*)status == 0 && sbase && (unsigned long long)sbase[nv] <= stage_slots);
    if (*(volatile const int*)status != 0) return;
    const unsigned lane = lane_id();
    const int64_t nth = (int64_t)gridDim.x * blockDim.x;
    for (int64_t b = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) & ~31ll; b < nv; b += nth) {
        const int64_t v = nv - 1 - (b + lane);  // from the top rank down
        int n = 0;
        if (v >= 0) {
            const int64_t dout = rp[v + 1] - rp[v], din = cp[v + 1] - cp[v];
            if (dout > 0 && din > 0 && is_block_row(dout, din, warp_cap, light_in)) n = (int)((din + kPart - 1) / kPart);
        }
        if (__ballot_sync(kFull, n > 0) == 0) continue;
        const int incl = warp_incl_scan(n);
        unsigned long long at = 0;
        if (lane == 31) at = atomicAdd(&ctl->nunits, (unsigned long long)incl);
        at = __shfl_sync(kFull, at, 31) + (unsigned long long)(incl - n);
        for (int i = 0; i < n; i++) units[at + i] = make_int2((int)v, i);
        if (n > 1) hubs[atomicAdd(&ctl->nhubs, 1ull)] = (int32_t)v;
    }
}

// A staged row (or column chunk of one): entries cols[e0, e0 + d).
struct WalkRow {
    uint32_t* bm;               // (set bits of the words before) << 16 | 16 bits
    uint32_t* cnt;              // kWalkCount: role-C counts
    uint8_t* perm;              // light rows wider than the bitmap: entry of the row by rank (block rows: null)
    int64_t e0;
    int d;
    int32_t wb;                 // first id
    uint32_t span;              // last id - first id
    uint32_t mask;
    bool exact;                 // span + 1 fits the bitmap (bit span + 1 stays clear: ids outside the row go there)
    uint32_t limit;             // entries of the longest tail that is streamed through it
    bool parts;                 // other units walk this row too
    bool chunked, more;         // the row is walked in column chunks; this is not its first
};

// A tail may be far longer than the row it is streamed through: v of few
// out-edges behind a source u of many, as in orders that are not degree ranks (the
// wheel of 200 K vertices with its hub at id 0 streams 20 G entries, 28 ms of
// support phase).  Past kLongTail entries and kLongRatio times the row's, the
// row's entries are searched in the tail instead (that wheel: 0.12 ms), so the
// walk stays within a factor of the rows' lengths.  Support phase streaming all
// of a tail / with ratios 32, 8 and 4: R-MAT scale 16 in id order 2.8 / 2.2, 1.6,
// 1.3 ms, with a hub joined to all of it 7.1 / 2.4, 1.7, 1.4; scale 18 in id
// order 35 / 26, 22, 21.  Tails of 512 instead of 128: a complete bipartite
// graph of 2 x 3,000 with a path on one side 2.8 instead of 1.9 (all streamed 2.8).  Degree
// ranks do not notice: scale 18 0.65 with any, scale 21 and 512 Barabasi-Albert
// graphs within 1 %.
constexpr uint32_t kLongTail = 128, kLongRatio = 4;
__device__ __forceinline__ uint32_t tail_limit(uint32_t dout) {
    return dout > UINT32_MAX / kLongRatio ? UINT32_MAX : max(kLongTail, kLongRatio * dout);
}

__device__ __forceinline__ WalkRow row_init(const WalkArgs& A, unsigned char* bm, unsigned char* cnt,
                                            unsigned char* perm, int log2bits, int64_t e0, int d, int64_t dout,
                                            bool more, bool parts) {
    WalkRow R;
    R.limit = tail_limit((uint32_t)dout);
    R.bm = reinterpret_cast<uint32_t*>(bm);
    R.cnt = reinterpret_cast<uint32_t*>(cnt);
    R.perm = perm;
    R.e0 = e0;
    R.d = d;
    R.wb = __ldg(A.cols + e0);
    R.span = (uint32_t)(__ldg(A.cols + e0 + d - 1) - R.wb);
    R.mask = (1u << log2bits) - 1u;
    R.exact = R.span < R.mask;
    R.chunked = dout > d;
    R.more = more;
    R.parts = parts;
    return R;
}

// Words of the bitmap in use.
__device__ __forceinline__ int row_words(const WalkRow& R) {
    return (int)((R.exact ? R.span + 1u : R.mask) >> 4) + 1;
}

// Sets the row's bits and its counters (the bitmap is clear).
__device__ __forceinline__ void row_fill(const WalkArgs& A, const WalkRow& R, int tid, int nthr) {
    for (int i = tid; i < R.d; i += nthr) {
        const int64_t e = R.e0 + i;
        const uint32_t x = (uint32_t)(__ldg(A.cols + e) - R.wb) & R.mask;
        atomicOr(R.bm + (x >> 4), 1u << (x & 15u));
        R.cnt[i] = 0u;
    }
}

// Rank of bit x in its word's terms: set bits of the row below it.
__device__ __forceinline__ int word_rank(uint32_t word, uint32_t x) {
    return (int)(word >> 16) + __popc(word & ((1u << (x & 15u)) - 1u));
}

// Position of id w in a row wider than the bitmap, when its bit is set (-1:
// another id's bit).
__device__ __forceinline__ int row_find(const WalkArgs& A, const WalkRow& R, uint32_t word, uint32_t x, int32_t w) {
    if (R.perm) {
        const int p = R.perm[word_rank(word, x)];
        if (__ldg(A.cols + R.e0 + p) == w) return p;
    }
    const int64_t p = find_sorted<int64_t>(A.cols, R.e0, R.e0 + R.d, w);
    return p < 0 ? -1 : (int)(p - R.e0);
}

constexpr uint32_t kNoEdge = UINT32_MAX;

// This warp's group of up to 32 in-edges.
struct WalkGroup {
    uint32_t* longs;            // per lane: its last in-edge with a long tail (kNoEdge: none)
    int4* ge;                   // per non-empty tail: {first chunk, begin, end, 0} (positions in colsA)
    int64_t* off;               // listing: slot of the in-edge's first role-A entry
    uint32_t* cnt;              // role-A entries found (listing: starts at the entries of earlier chunks)
};

// First slot of the role-A entries of in-edge eid, an edge of row u = [beg, end).
template <int M>
__device__ __forceinline__ int64_t role_a_slot(const WalkArgs& A, int32_t eid, int32_t u, int64_t beg, int64_t end) {
    return M == kWalkList ? __ldg(A.off + eid) : stage_slot(__ldg(A.sbase + u), end - beg, eid - beg);
}

// Role-A entries of an in-edge found so far (all of them unless its row is
// walked in chunks).
template <int M>
__device__ __forceinline__ void role_a_done(const WalkArgs& A, int32_t eid, uint32_t c, bool chunked) {
    if (chunked) A.runA[eid] = (int32_t)c;
    if (M == kWalkCount) A.cA[eid] = (int32_t)c;
    else if (!chunked && c != (uint32_t)__ldg(A.cA + eid)) atomicMax(A.status, (int)TDT_ERR_CAPACITY);
}

// The in-edges with long tails that each lane of a warp left for the end of the
// warp's work, a list through longs from the last one.  The entries of their
// rows N+(v), of 32 in-edges (u,v) as one flat space, are searched in the tails.
// The rows' own counts have been flushed by this block.  (Searched on the spot they
// cost the walk of 512 Barabasi-Albert graphs 8 %: registers around a call that
// never came.)
template <int M>
__device__ __forceinline__ void walk_long_tails(const WalkArgs& A, const WalkGroup& Q, bool list, int2* out0,
                                                int64_t cap) {
    const unsigned lane = lane_id();
    __syncwarp();
    uint32_t k = Q.longs[lane];
    Q.longs[lane] = kNoEdge;
    while (__any_sync(kFull, k != kNoEdge)) {
        int32_t eid = 0;
        uint32_t n = 0;
        int64_t end = 0, e0 = 0;
        const bool mine = k != kNoEdge;
        if (mine) {
            const int32_t u = __ldg(A.in_src + k);
            eid = __ldg(A.in_eid + k);
            k = A.longs[k];
            const int32_t v = __ldg(A.cols + eid);
            e0 = __ldg(A.rp + v);
            n = (uint32_t)(__ldg(A.rp + v + 1) - e0);
            end = __ldg(A.rp + u + 1);
            if (list) Q.off[lane] = role_a_slot<M>(A, eid, u, __ldg(A.rp + u), end);
            Q.cnt[lane] = 0u;
        }
        __syncwarp();
        // 32 pairs (u,v) that differ, and rows a quarter of their tails at most: less
        // than 1.4 E in all, which 32 bits hold
        const uint32_t incl = warp_incl_scan(n);
        const uint32_t total = __shfl_sync(kFull, incl, 31), S = incl - n;
        for (uint32_t b = 0; b < total; b += kWarp) {
            const uint32_t at = b + lane;
            int own = 0;  // last lane with S <= at
#pragma unroll
            for (int step = 16; step > 0; step >>= 1)
                if (__shfl_sync(kFull, S, own + step) <= at) own += step;
            const int64_t e = __shfl_sync(kFull, e0, own) + (at - __shfl_sync(kFull, S, own));
            const int64_t lo = (int64_t)__shfl_sync(kFull, eid, own) + 1, hi = __shfl_sync(kFull, end, own);
            if (at >= total) continue;
            const int64_t p = find_sorted<int64_t>(A.cols, lo, hi, __ldg(A.cols + e));
            if (p < 0) continue;
            if (M == kWalkCount) {
                atomicAdd(A.cB + p, 1);
                atomicAdd(A.cC + e, 1);
            }
            const uint32_t old = atomicAdd(Q.cnt + own, 1u);
            if (list) {
                const int64_t to = Q.off[own] + old;
                if (to < cap) out0[to] = make_int2((int32_t)p, (int32_t)e);
            }
        }
        __syncwarp();
        if (mine) role_a_done<M>(A, eid, Q.cnt[lane], false);
        __syncwarp();
    }
}

// One in-edge per lane, at position k of the in-adjacency (k < 0: none), of
// the staged row or, Kind = kRowTiny, each of its own row cols[e0, e0 + d).
// list: role-A entries are stored (A.out is indexed forward from out0, stores
// stay below cap).
enum RowKind { kRowExact = 0, kRowHashed = 1, kRowTiny = 2 };

template <int M, int Kind>
__device__ __forceinline__ void walk_in_edges(const WalkArgs& A, const WalkRow& R, const WalkGroup& Q,
                                              const int4* __restrict__ cols4, unsigned sh, bool list, int2* out0,
                                              int64_t cap, int64_t k, int64_t e0, int d) {
    const unsigned lane = lane_id();
    const unsigned lt = lanemask_lt(), le = lt | (1u << lane);
    constexpr bool Exact = Kind == kRowExact;
    int32_t eid = 0, units = 0;
    unsigned lo = 0, hi = 0;
    int64_t slot = 0;
    if (k >= 0) {
        const int32_t u = __ldg(A.in_src + k);
        eid = __ldg(A.in_eid + k);
        const int64_t end = __ldg(A.rp + u + 1);
        lo = (unsigned)eid + 1u + sh;
        hi = (unsigned)end + sh;
        if (hi > lo) {
            if (hi - lo <= (Kind == kRowTiny ? tail_limit((uint32_t)d) : R.limit)) {
                units = (int32_t)(((hi + 3u) >> 2) - (lo >> 2));
                if (list) slot = role_a_slot<M>(A, eid, u, __ldg(A.rp + u), end);
            } else if (Kind == kRowTiny || !R.more) {
                A.longs[k] = Q.longs[lane];
                Q.longs[lane] = (uint32_t)k;
            }
        }
    }
    const unsigned nem = __ballot_sync(kFull, units > 0);
    if (nem == 0) return;
    const int n = __popc(nem);
    const int32_t incl = warp_incl_scan(units);
    const int32_t total = __shfl_sync(kFull, incl, 31);
    const int ci = __popc(nem & lt);
    if (units > 0) {
        Q.ge[ci] = make_int4(incl - units, (int)lo, (int)hi, (int)lane);
        if (list) Q.off[ci] = slot;
        Q.cnt[ci] = Kind != kRowTiny && R.more ? (uint32_t)A.runA[eid] : 0u;
    }
    __syncwarp();
    uint32_t wb = 0, over = 0, mask = 0;
    if (Kind != kRowTiny) {
        wb = (uint32_t)R.wb;
        over = R.span + 1u;
        mask = R.mask;
    }
    int ob = 0;
    for (int base = 0; base < total; base += kWarp) {
        // tails that start inside (base, base + 32): each is > base, at most 31 fit
        const int kk = ob + 1 + (int)lane;
        const int32_t B = kk < n ? Q.ge[kk].x : INT32_MAX;
        const unsigned bit = ((unsigned)(B - base) < (unsigned)kWarp) ? (1u << (B - base)) : 0u;
        const unsigned mk = __reduce_or_sync(kFull, bit);
        const int nb = __popc(mk);
        const int32_t Bn = __shfl_sync(kFull, B, nb);
        const int c = base + (int)lane;
        const int o = ob + __popc(mk & le);
        const int4 ge = Q.ge[o];
        const unsigned glo = (unsigned)ge.y, ghi = (unsigned)ge.z;
        const unsigned p0 = ((glo >> 2) + (unsigned)(c - ge.x)) << 2;
        unsigned cm = 0;  // entries inside [glo, ghi)
        int4 w4 = make_int4(0, 0, 0, 0);
        if (c < total) {
            w4 = __ldg(cols4 + (p0 >> 2));
            cm = 0xFu;
            if (p0 < glo) cm &= 0xFu << (glo - p0);
            if (p0 + 4u > ghi) cm &= 0xFu >> (p0 + 4u - ghi);
        }
        const int32_t w[4] = {w4.x, w4.y, w4.z, w4.w};
        bool hit[4];
        int p[4];
        int64_t row0 = 0;  // first edge of the row the hits are in
        uint32_t x[4], word[4];
        if (Kind == kRowTiny) {
            row0 = __shfl_sync(kFull, e0, ge.w);
            const int dr = __shfl_sync(kFull, d, ge.w);
            // four searches in step: the last entry <= w
            const int32_t* row = A.cols + row0;
#pragma unroll
            for (int q = 0; q < 4; q++) p[q] = 0;
            for (int s = dr > 1 ? 1 << (31 - __clz(dr - 1)) : 0; s > 0; s >>= 1) {
#pragma unroll
                for (int q = 0; q < 4; q++)
                    if (p[q] + s < dr && __ldg(row + p[q] + s) <= w[q]) p[q] += s;
            }
#pragma unroll
            for (int q = 0; q < 4; q++) hit[q] = ((cm >> q) & 1u) != 0u && __ldg(row + p[q]) == w[q];
        } else {
            row0 = R.e0;
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const uint32_t dw = (uint32_t)w[q] - wb;
                x[q] = Exact ? min(dw, over) : dw & mask;
                word[q] = R.bm[x[q] >> 4];
            }
#pragma unroll
            for (int q = 0; q < 4; q++) {
                hit[q] = ((word[q] >> (x[q] & 15u)) & (cm >> q) & 1u) != 0u;
                p[q] = Exact ? word_rank(word[q], x[q]) : -1;
            }
        }
        if (Kind == kRowHashed) {
#pragma unroll
            for (int q = 0; q < 4; q++) {
                if (hit[q]) p[q] = row_find(A, R, word[q], x[q], w[q]);
                hit[q] = p[q] >= 0;
            }
        }
        const int64_t pos = (int64_t)p0 - sh;
        if (M == kWalkCount) {
            int32_t* cb = A.cB + pos;
#pragma unroll
            for (int q = 0; q < 4; q++) {
                if (hit[q]) {
                    if (Kind == kRowTiny) atomicAdd(A.cC + row0 + p[q], 1);
                    else atomicAdd(R.cnt + p[q], 1u);
                }
                if (hit[q]) atomicAdd(cb + q, 1);
            }
        }
        // this lane's tail within the step: lanes [first, next) from the starts
        const unsigned st = mk | 1u;
        const int first = 31 - __clz(st & le);
        const unsigned after = st & ~le;
        const unsigned seg = ((after & (0u - after)) - 1u) & (0xffffffffu << first);
        unsigned m[4];
        int na = 0;
#pragma unroll
        for (int q = 0; q < 4; q++) {
            m[q] = __ballot_sync(kFull, hit[q]) & seg;
            na += __popc(m[q]);
        }
        uint32_t old = 0;
        if ((int)lane == first && na) {
            old = Q.cnt[o];
            Q.cnt[o] = old + (uint32_t)na;
        }
        if (list) {
            old = __shfl_sync(kFull, old, first);
            int64_t s = Q.off[o] + old;
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int64_t at = s + __popc(m[q] & lt);
                if (hit[q] && at < cap) out0[at] = make_int2((int32_t)pos + q, (int32_t)(row0 + p[q]));
                s += __popc(m[q]);
            }
        }
        ob += nb + (Bn == base + kWarp ? 1 : 0);
        __syncwarp();
    }
    if (units > 0) role_a_done<M>(A, eid, Q.cnt[ci], Kind != kRowTiny && R.chunked);
    __syncwarp();
}

// Role-C counts of the row to global memory.
__device__ __forceinline__ void row_flush(const WalkArgs& A, const WalkRow& R, int tid, int nthr) {
    for (int i = tid; i < R.d; i += nthr) {
        const uint32_t c = R.cnt[i];
        if (c == 0) continue;
        if (R.parts) atomicAdd(A.cC + R.e0 + i, (int32_t)c);
        else A.cC[R.e0 + i] = (int32_t)c;
    }
}

template <int M>
__global__ void __launch_bounds__(kWkBlock, kWkMinBlocks) walk_kernel(const __grid_constant__ WalkArgs A,
                                                                      WalkCtl* ctl, int light_batch) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int s_wsum[kWkWarps];
    __shared__ unsigned long long s_unit;
    __shared__ int s_next;
    __shared__ uint32_t s_longs[kWkBlock];
    const bool failed = M == kWalkList && look_back_failed(A.status);  // the offsets are not the scan's
    if ((A.gate && *(volatile const int*)A.gate != 0) || failed) return;
    const int wib = threadIdx.x / kWarp;
    const unsigned lane = lane_id();
    const unsigned sh = (unsigned)(((uintptr_t)A.cols & 15u) >> 2);
    const int4* cols4 = reinterpret_cast<const int4*>(A.cols - sh);
    // listing: the staging slots end at A.out, the lists start there
    const bool list = M == kWalkList || (A.sbase && *(volatile const int*)A.stage_skip == 0);
    const int64_t cap = !list ? 0 : M == kWalkList ? __ldg(A.off + A.ne) : __ldg(A.sbase + A.nv);
    int2* out0 = M == kWalkList ? A.out : A.out - cap;
    unsigned char* gs = smem + kWkRowBytes + wib * kGrpBytes;
    WalkGroup Q;
    Q.longs = s_longs + wib * kWarp;
    Q.ge = reinterpret_cast<int4*>(gs);
    Q.off = reinterpret_cast<int64_t*>(gs + 16 * kWarp);
    Q.cnt = reinterpret_cast<uint32_t*>(gs + 24 * kWarp);

    Q.longs[lane] = kNoEdge;

    // ---- block rows, a unit a turn, and the warp rows in the last one.  Each turn
    // ends with the searches it left: a block that only left them would take the
    // most units.
    const unsigned long long nunits = ctl->nunits;
    for (;;) {
        if (threadIdx.x == 0) s_unit = atomicAdd(&ctl->unit_next[M], 1ull);
        __syncthreads();
        const unsigned long long ui = s_unit;
        const bool last = ui >= nunits;
        if (!last) {
            const int2 un = __ldg(A.units + ui);
            const int64_t v = un.x;
            const int64_t r0 = __ldg(A.rp + v), r1 = __ldg(A.rp + v + 1);
            const int64_t i0 = __ldg(A.cp + v), i1 = __ldg(A.cp + v + 1);
            const int64_t ka = i0 + (int64_t)un.y * kPart, kb = ka + kPart < i1 ? ka + kPart : i1;
            const bool parts = i1 - i0 > kPart;
            for (int64_t c0 = r0; c0 < r1; c0 += A.row_cap) {
                const int d = (int)(r1 - c0 < A.row_cap ? r1 - c0 : A.row_cap);
                WalkRow R = row_init(A, smem + kWkBm, smem + kWkCnt, nullptr, kHeavyLog2, c0, d, r1 - r0, c0 > r0, parts);
                const int nw = row_words(R);
                for (int i = threadIdx.x; i < nw; i += kWkBlock) R.bm[i] = 0u;
                if (threadIdx.x == 0) s_next = 0;
                __syncthreads();
                row_fill(A, R, threadIdx.x, kWkBlock);
                __syncthreads();
                if (R.exact) {
                    // running counts: each thread's run of words, then a block scan
                    const int per = (nw + kWkBlock - 1) / kWkBlock;
                    const int a = threadIdx.x * per, b = a + per < nw ? a + per : nw;
                    int s = 0;
                    for (int i = a; i < b; i++) s += __popc(R.bm[i]);
                    const int incl = warp_incl_scan(s);
                    if (lane == 31) s_wsum[wib] = incl;
                    __syncthreads();
                    int run = incl - s;
                    for (int i = 0; i < wib; i++) run += s_wsum[i];
                    for (int i = a; i < b; i++) {
                        const uint32_t word = R.bm[i];
                        R.bm[i] = word | ((uint32_t)run << 16);
                        run += __popc(word);
                    }
                    __syncthreads();
                }
                for (;;) {
                    int nx = 0;
                    if (lane == 0) nx = atomicAdd(&s_next, kWarp);
                    nx = __shfl_sync(kFull, nx, 0);
                    if (ka + nx >= kb) break;
                    const int64_t k = ka + nx + lane < kb ? ka + nx + lane : -1;
                    if (R.exact) walk_in_edges<M, kRowExact>(A, R, Q, cols4, sh, list, out0, cap, k, 0, 0);
                    else walk_in_edges<M, kRowHashed>(A, R, Q, cols4, sh, list, out0, cap, k, 0, 0);
                }
                __syncthreads();
                if (M == kWalkCount) row_flush(A, R, threadIdx.x, kWkBlock);
                __syncthreads();
            }
        } else {
            // ---- warp rows from the top rank down, one lane per row finding those
            // with work: two at a time in the top quarter, where most of the work is
            // (a long batch there left one warp running alone), then light_batch
            const unsigned long long t1 = ((unsigned long long)A.nv + 3) / 4;
            unsigned char* sl = smem + wib * kLtBytes;
            for (;;) {
                unsigned long long t = 0;
                if (lane == 0) t = atomicAdd(&ctl->light_next[M], 1ull);
                t = __shfl_sync(kFull, t, 0);
                const unsigned long long g1 = (t1 + kTopBatch - 1) / kTopBatch;
                const int batch = t < g1 ? kTopBatch : light_batch;
                const unsigned long long first = t < g1 ? t * kTopBatch : g1 * kTopBatch + (t - g1) * (unsigned)light_batch;
                if (first >= (unsigned long long)A.nv) break;
                const int64_t mine = A.nv - 1 - (int64_t)first - (int64_t)lane;
                int64_t r0 = 0, i0 = 0;
                int d = 0, din = 0;
                if ((int)lane < batch && mine >= 0) {
                    r0 = __ldg(A.rp + mine);
                    i0 = __ldg(A.cp + mine);
                    const int64_t dout = __ldg(A.rp + mine + 1) - r0, di = __ldg(A.cp + mine + 1) - i0;
                    if (dout > 0 && di > 0 && !is_block_row(dout, di, A.warp_cap, A.light_in)) {
                        d = (int)dout;
                        din = (int)di;
                    }
                }
                // tiny rows: their in-edges, 32 at a time
                const bool tiny = d > 0 && is_tiny_row(d, din);
                if (__ballot_sync(kFull, tiny)) {
                    const int tn = tiny ? din : 0;
                    const int tincl = warp_incl_scan(tn);
                    const int ttotal = __shfl_sync(kFull, tincl, 31);
                    const int ts = tincl - tn;
                    for (int b = 0; b < ttotal; b += kWarp) {
                        const int at = b + (int)lane;
                        int own = 0;  // last lane with ts <= at
        #pragma unroll
                        for (int step = 16; step > 0; step >>= 1)
                            if (__shfl_sync(kFull, ts, own + step) <= at) own += step;
                        const int64_t k = __shfl_sync(kFull, i0, own) + (at - __shfl_sync(kFull, ts, own));
                        const int64_t e0 = __shfl_sync(kFull, r0, own);
                        const int dr = __shfl_sync(kFull, d, own);
                        walk_in_edges<M, kRowTiny>(A, WalkRow{}, Q, cols4, sh, list, out0, cap, at < ttotal ? k : -1, e0, dr);
                    }
                }
                unsigned todo = __ballot_sync(kFull, d > 0 && !tiny);
                while (todo) {
                    const int src = __ffs(todo) - 1;
                    todo &= todo - 1;
                    const int64_t e0 = __shfl_sync(kFull, r0, src), k0 = __shfl_sync(kFull, i0, src);
                    const int dr = __shfl_sync(kFull, d, src), dk = __shfl_sync(kFull, din, src);
                    WalkRow R = row_init(A, sl + kLtBm, sl + kLtCnt, sl + kLtPerm, kLightLog2, e0, dr, dr, false, false);
                    const int nw = row_words(R);
                    for (int i = lane; i < nw; i += kWarp) R.bm[i] = 0u;
                    __syncwarp();
                    row_fill(A, R, lane, kWarp);
                    __syncwarp();
                    int run = 0;
                    for (int b = 0; b < nw; b += kWarp) {
                        const int i = b + (int)lane;
                        const uint32_t word = i < nw ? R.bm[i] : 0u;
                        const int s = __popc(word);
                        const int incl = warp_incl_scan(s);
                        if (i < nw) R.bm[i] = word | ((uint32_t)(run + incl - s) << 16);
                        run += __shfl_sync(kFull, incl, 31);
                    }
                    __syncwarp();
                    if (R.exact) {
                        for (int k = lane; k - (int)lane < dk; k += kWarp)
                            walk_in_edges<M, kRowExact>(A, R, Q, cols4, sh, list, out0, cap, k < dk ? k0 + k : -1, 0, 0);
                    } else {
                        for (int i = lane; i < dr; i += kWarp) {
                            const uint32_t x = (uint32_t)(__ldg(A.cols + e0 + i) - R.wb) & R.mask;
                            R.perm[word_rank(R.bm[x >> 4], x)] = (uint8_t)i;
                        }
                        __syncwarp();
                        for (int k = lane; k - (int)lane < dk; k += kWarp)
                            walk_in_edges<M, kRowHashed>(A, R, Q, cols4, sh, list, out0, cap, k < dk ? k0 + k : -1, 0, 0);
                    }
                    if (M == kWalkCount) row_flush(A, R, lane, kWarp);
                    __syncwarp();
                }
            }
        }
        walk_long_tails<M>(A, Q, list, out0, cap);
        if (last) break;
    }
}

// Roles B and C from the role-A entries (eB, eC) of eA = (u,v):
//   role B: eB gets (eA, eC); sources and targets are edges of the same row;
//   role C: eC gets (eA, eB); sources are the in-edges of v, targets its
//           out-edges.
// Sources are taken in order (edges, or in-edges grouped by v) in windows
// rounded to whole rows (whole v's), so a window owns its targets and keeps
// their slot cursors.  The in-edges of a hub, a v of more than kPart, are
// spread over windows: each chunk then reserves the runs of the hub's targets
// with one global atomic per run.  Lists of few entries get wider windows
// (each costs a chain of dependent loads), and below kDsSparse entries a list
// there is nothing to sort: a warp takes 32 sources and stores entry by entry,
// a global atomic each (512 Barabasi-Albert graphs, 0.3 triangles an edge:
// 1.7 ms of listing in windows).
// A window's entries pass through chunks of kDsChunk: ranks
// among equal targets from shared-memory counters, the chunk laid out by
// target in shared memory, then written out by consecutive threads, a run per
// target.  A window with more than kDsKeys targets (or lists past 32-bit
// offsets) stores entry by entry with cursors in global memory.  Role B also
// moves the role-A entries from their staging slots to the lists.  Every
// cursor must end where the next role's entries begin.
constexpr int kDsBlock = 256;
constexpr int kDsWarps = kDsBlock / kWarp;
constexpr int kDsPer = 8;              // entries per thread and chunk
constexpr int kDsChunk = kDsBlock * kDsPer;
constexpr int kDsWinMin = 256, kDsWinMax = 1024;
constexpr int kDsWinEntries = 4096;             // entries of a window aimed at, at the lists' mean length
constexpr int kDsSparse = 2;
constexpr int kDsKeys = 2048;
static_assert(kPart >= kDsWinMax, "a hub lies at an end of its windows");
static_assert(kDsKeys <= 65536 && kDsChunk <= 65536, "16-bit keys");

struct DistArgs {
    const int64_t* rp;
    const int32_t* cols;
    const int32_t* rows;
    const int64_t* cp;
    const int32_t* in_eid;
    int64_t nv, ne;
    const int64_t* off;
    const int32_t* cA;
    const int32_t* cB;
    const int64_t* sbase;       // role B: staging slots before each row
    const int2* stage_end;      // role B: end of the staging slots
    const int* stage_skip;      // role B: non-zero: the role-A entries are in the lists already
    int2* lists;
    uint32_t* cnt;              // entries stored one by one, and of hubs (zero before role B; see below)
    const int32_t* hubs;        // of the walk's plan
    int* status;
    const int* gate;
};

constexpr int kDsCnt = 0;
constexpr int kDsCur = kDsCnt + 4 * kDsKeys;
constexpr int kDsDst = kDsCur + 4 * kDsKeys;
constexpr int kDsBuf = kDsDst + 4 * kDsKeys;
constexpr int kDsKey = kDsBuf + 8 * kDsChunk;
constexpr int kDsSmem = kDsKey + 2 * kDsChunk;

template <bool RoleC>
__global__ void __launch_bounds__(kDsBlock, 4) distribute_kernel(const __grid_constant__ DistArgs A,
                                                                           WalkCtl* ctl) {
    extern __shared__ __align__(16) unsigned char smem[];
    uint32_t* s_cnt = reinterpret_cast<uint32_t*>(smem + kDsCnt);  // per target: chunk count, then its start in the chunk
    uint32_t* s_cur = reinterpret_cast<uint32_t*>(smem + kDsCur);  // slots written so far, relative to base
    uint32_t* s_dst = reinterpret_cast<uint32_t*>(smem + kDsDst);  // slot of the run minus its start in the chunk
    int2* s_buf = reinterpret_cast<int2*>(smem + kDsBuf);
    uint16_t* s_key = reinterpret_cast<uint16_t*>(smem + kDsKey);
    __shared__ int32_t s_S[kDsBlock];
    __shared__ int32_t s_E[kDsBlock];
    __shared__ int64_t s_O[kDsBlock];
    __shared__ int64_t s_F[RoleC ? 1 : kDsBlock];  // role B: where the staged role-A entries go
    __shared__ int32_t s_wsum[2][kDsWarps];
    __shared__ unsigned long long s_win;
    const bool failed = look_back_failed(A.status);  // the offsets are not the scan's
    if ((A.gate && *(volatile const int*)A.gate != 0) || failed) return;
    const int wib = threadIdx.x / kWarp;
    const unsigned lane = lane_id();
    const unsigned lt = lanemask_lt(), le = lt | (1u << lane);
    const bool staged = !RoleC && *(volatile const int*)A.stage_skip == 0;
    const int2* src = staged ? A.stage_end - __ldg(A.sbase + A.nv) : A.lists;
    const unsigned long long cap = (unsigned long long)__ldg(A.off + A.ne);
    int64_t win = kDsWinMax;
    while (win > kDsWinMin && (int64_t)(cap / 3) * win > A.ne * kDsWinEntries) win >>= 1;
    while (win > 32 && A.ne < win * 2 * gridDim.x) win >>= 1;  // small graphs: two windows a block
    const int64_t nwin = (A.ne + win - 1) / win;
    // first source at or after position p that starts a row (role C: a v)
    auto first_source = [&](int64_t p) -> int64_t {
        if (p >= A.ne) return A.ne;
        const int64_t* ptr = RoleC ? A.cp : A.rp;
        const int32_t x = RoleC ? __ldg(A.cols + __ldg(A.in_eid + p)) : __ldg(A.rows + p);
        const int64_t s = __ldg(ptr + x), t = __ldg(ptr + x + 1);
        return s == p || (RoleC && t - s > kPart) ? p : t;
    };
    auto staged_at = [&](int32_t e) -> int64_t {
        const int32_t u = __ldg(A.rows + e);
        const int64_t r0 = __ldg(A.rp + u);
        return stage_slot(__ldg(A.sbase + u), __ldg(A.rp + u + 1) - r0, e - r0);
    };
    auto hub_rows = [&](unsigned long long first, unsigned long long step, auto&& f) {  // f(edge) over the hubs' out-edges
        for (unsigned long long i = first; i < ctl->nhubs; i += step) {
            const int32_t v = __ldg(A.hubs + i);
            for (int64_t e = __ldg(A.rp + v) + threadIdx.x; e < __ldg(A.rp + v + 1); e += kDsBlock) f(e);
        }
    };
    if (cap < (unsigned long long)A.ne * 3 * kDsSparse) {
        // cnt counts on from role B to role C
        const int64_t nwarps = (int64_t)gridDim.x * kDsWarps;
        for (int64_t k0 = ((int64_t)blockIdx.x * kDsWarps + wib) * kWarp; k0 < A.ne; k0 += nwarps * kWarp) {
            const int64_t k = k0 + lane;
            int32_t e = 0, len = 0;
            if (k < A.ne) {
                e = RoleC ? __ldg(A.in_eid + k) : (int32_t)k;
                len = __ldg(A.cA + e);
            }
            const int32_t incl = warp_incl_scan(len);
            const int32_t total = __shfl_sync(kFull, incl, 31);
            if (total == 0) continue;
            const int32_t S = incl - len;
            int64_t o = 0, f = 0;
            if (len) {
                o = f = __ldg(A.off + e);
                if (staged) o = staged_at(e);
            }
            for (int32_t b = 0; b < total; b += kWarp) {
                const int32_t t = b + (int)lane;
                int own = 0;  // last lane with S <= t
#pragma unroll
                for (int step = 16; step > 0; step >>= 1)
                    if (__shfl_sync(kFull, S, own + step) <= t) own += step;
                const int32_t at = t - __shfl_sync(kFull, S, own);
                const int64_t os = __shfl_sync(kFull, o, own), fs = __shfl_sync(kFull, f, own);
                const int32_t eA = __shfl_sync(kFull, e, own);
                if (t >= total) continue;
                const int2 ent = __ldcg(src + os + at);  // (eB, eC)
                if (!RoleC && staged && (unsigned long long)(fs + at) < cap) A.lists[fs + at] = ent;
                const int32_t x = RoleC ? ent.y : ent.x;
                if (x < 0 || x >= A.ne) {
                    atomicMax(A.status, (int)TDT_ERR_CAPACITY);
                    continue;
                }
                const unsigned long long to =
                    (unsigned long long)(__ldg(A.off + x) + __ldg(A.cA + x)) + atomicAdd(A.cnt + x, 1u);
                if (to < cap) A.lists[to] = make_int2(eA, RoleC ? ent.x : ent.y);
            }
        }
        return;
    }
    for (int i = threadIdx.x; i < kDsKeys; i += kDsBlock) s_cnt[i] = 0u;
    for (;;) {
        if (threadIdx.x == 0) s_win = atomicAdd(&ctl->dist_next[RoleC ? 1 : 0], 1ull);
        __syncthreads();
        // from the top rank down: the windows of hubs first
        const int64_t wi = nwin - 1 - (int64_t)s_win;
        if (wi < 0) break;
        const int64_t ka = first_source(wi * win), kb = first_source((wi + 1) * win);
        if (ka >= kb) {
            __syncthreads();
            continue;
        }
        // target edges [ta, tb); those below own0 or from own1 on are a hub's
        int64_t ta = ka, tb = kb, own0 = ka, own1 = kb;
        if (RoleC) {
            const int32_t va = __ldg(A.cols + __ldg(A.in_eid + ka)), vb = __ldg(A.cols + __ldg(A.in_eid + kb - 1));
            ta = own0 = __ldg(A.rp + va);
            tb = own1 = __ldg(A.rp + vb + 1);
            if (__ldg(A.cp + va + 1) - __ldg(A.cp + va) > kPart) own0 = __ldg(A.rp + va + 1);
            if (__ldg(A.cp + vb + 1) - __ldg(A.cp + vb) > kPart) own1 = __ldg(A.rp + vb);
        }
        const int64_t base = __ldg(A.off + ta);
        const bool keyed = tb - ta <= kDsKeys && __ldg(A.off + tb) - base < (1ll << 32);
        const int nkeys = keyed ? (int)(tb - ta) : 0;
        // first slot of a target's entries of this role
        auto first_slot = [&](int64_t e) { return __ldg(A.off + e) + __ldg(A.cA + e) + (RoleC ? __ldg(A.cB + e) : 0); };
        if (keyed)
            for (int64_t e = ta + threadIdx.x; e < tb; e += kDsBlock) s_cur[e - ta] = (uint32_t)(first_slot(e) - base);
        __syncthreads();
        for (int64_t g0 = ka; g0 < kb; g0 += kDsBlock) {
            // the role-A entries of 256 sources as one flat space
            const int64_t k = g0 + threadIdx.x;
            int32_t e = 0, len = 0;
            if (k < kb) {
                e = RoleC ? __ldg(A.in_eid + k) : (int32_t)k;
                len = __ldg(A.cA + e);
            }
            const unsigned nem = __ballot_sync(kFull, len > 0);
            const int32_t incl = warp_incl_scan(len);
            if (lane == 31) {
                s_wsum[0][wib] = incl;
                s_wsum[1][wib] = __popc(nem);
            }
            __syncthreads();
            int32_t S = incl - len, total = 0;
            int ci = __popc(nem & lt), n = 0;
#pragma unroll
            for (int w = 0; w < kDsWarps; w++) {
                if (w < wib) {
                    S += s_wsum[0][w];
                    ci += s_wsum[1][w];
                }
                total += s_wsum[0][w];
                n += s_wsum[1][w];
            }
            if (len > 0) {
                s_S[ci] = S;
                s_E[ci] = e;
                const int64_t o = __ldg(A.off + e);
                s_O[ci] = o;
                if (!RoleC && staged) {
                    s_O[ci] = staged_at(e);
                    s_F[ci] = o;
                }
            }
            __syncthreads();
            for (int cs = 0; cs < total; cs += kDsChunk) {
                const int ce = cs + kDsChunk < total ? cs + kDsChunk : total;
                int key[kDsPer];
                uint32_t rank[kDsPer];
                int2 ent[kDsPer];
                const int p0 = cs + wib * (kDsPer * kWarp);
#pragma unroll
                for (int h = 0; h < kDsPer; h++) key[h] = -1;
                if (p0 < ce) {
                    int ob = 0;
                    if (lane == 0) {
                        int lo = 0, hi = n - 1;  // last list with S <= p0
                        while (lo < hi) {
                            const int mid = (lo + hi + 1) >> 1;
                            if (s_S[mid] <= p0) lo = mid; else hi = mid - 1;
                        }
                        ob = lo;
                    }
                    ob = __shfl_sync(kFull, ob, 0);
                    int o[kDsPer];
#pragma unroll
                    for (int h = 0; h < kDsPer; h++) {
                        const int b = p0 + h * kWarp;
                        // list starts inside (b, b + 32): each is > b, at most 31 fit
                        const int kk = ob + 1 + (int)lane;
                        const int32_t B = kk < n ? s_S[kk] : INT32_MAX;
                        const unsigned bit = ((unsigned)(B - b) < (unsigned)kWarp) ? (1u << (B - b)) : 0u;
                        const unsigned mk = __reduce_or_sync(kFull, bit);
                        const int nb = __popc(mk);
                        const int32_t Bn = __shfl_sync(kFull, B, nb);
                        o[h] = ob + __popc(mk & le);
                        ent[h] = make_int2(-1, -1);
                        if (b + (int)lane < ce) {
                            const int64_t at = b + (int)lane - s_S[o[h]];
                            ent[h] = __ldcg(src + s_O[o[h]] + at);  // (eB, eC)
                        }
                        ob += nb + (Bn == b + kWarp ? 1 : 0);
                    }
#pragma unroll
                    for (int h = 0; h < kDsPer; h++) {
                        const int b = p0 + h * kWarp;
                        if (b + (int)lane >= ce) continue;
                        if (!RoleC && staged) {
                            const unsigned long long at = (unsigned long long)s_F[o[h]] + (b + (int)lane - s_S[o[h]]);
                            if (at < cap) A.lists[at] = ent[h];
                        }
                        const int64_t t = (int64_t)(RoleC ? ent[h].y : ent[h].x);
                        if (t < ta || t >= tb) {
                            atomicMax(A.status, (int)TDT_ERR_CAPACITY);
                            continue;
                        }
                        ent[h] = make_int2(s_E[o[h]], RoleC ? ent[h].x : ent[h].y);
                        if (keyed) {
                            key[h] = (int)(t - ta);
                            rank[h] = atomicAdd(s_cnt + key[h], 1u);
                        } else {
                            const unsigned long long at = (unsigned long long)first_slot(t) + atomicAdd(A.cnt + t, 1u);
                            if (at < cap) A.lists[at] = ent[h];
                        }
                    }
                }
                if (!keyed) continue;
                __syncthreads();
                if (RoleC && (own0 > ta || own1 < tb)) {
                    // a hub's runs, one thread per target
                    for (int i = threadIdx.x; i < nkeys; i += kDsBlock) {
                        const uint32_t c = s_cnt[i];
                        if (c && (ta + i < own0 || ta + i >= own1))
                            s_cur[i] = (uint32_t)(first_slot(ta + i) - base) + atomicAdd(A.cnt + ta + i, c);
                    }
                    __syncthreads();
                }
                {
                    // chunk starts of the targets; their runs' slots
                    const int per = (nkeys + kDsBlock - 1) / kDsBlock;
                    const int a = threadIdx.x * per, b = a + per < nkeys ? a + per : nkeys;
                    uint32_t s = 0;
                    for (int i = a; i < b; i++) s += s_cnt[i];
                    const uint32_t in = warp_incl_scan(s);
                    if (lane == 31) s_wsum[0][wib] = (int)in;
                    __syncthreads();
                    uint32_t run = in - s;
                    for (int w = 0; w < wib; w++) run += (uint32_t)s_wsum[0][w];
                    for (int i = a; i < b; i++) {
                        const uint32_t c = s_cnt[i], at = s_cur[i];
                        s_cnt[i] = run;
                        s_dst[i] = at - run;
                        s_cur[i] = at + c;
                        run += c;
                    }
                }
                __syncthreads();
#pragma unroll
                for (int h = 0; h < kDsPer; h++) {
                    if (key[h] < 0) continue;
                    const uint32_t at = s_cnt[key[h]] + rank[h];
                    s_buf[at] = ent[h];
                    s_key[at] = (uint16_t)key[h];
                }
                __syncthreads();
                for (int i = threadIdx.x; i < ce - cs; i += kDsBlock) {
                    const unsigned long long at =
                        (unsigned long long)base + (uint32_t)(s_dst[s_key[i]] + (uint32_t)i);
                    if (at < cap) A.lists[at] = s_buf[i];
                }
                for (int i = threadIdx.x; i < nkeys; i += kDsBlock) s_cnt[i] = 0u;
                __syncthreads();
            }
            __syncthreads();  // the group arrays are rewritten next
        }
        for (int64_t e = ta + threadIdx.x; e < tb; e += kDsBlock) {
            if (e < own0 || e >= own1) continue;
            const uint32_t want = (uint32_t)(RoleC ? __ldg(A.off + e + 1) - first_slot(e) : __ldg(A.cB + e));
            const uint32_t got = keyed ? s_cur[e - ta] - (uint32_t)(first_slot(e) - base) : __ldcg(A.cnt + e);
            if (got != want) atomicMax(A.status, (int)TDT_ERR_CAPACITY);
            if (!RoleC && !keyed) A.cnt[e] = 0u;  // role C counts from zero
        }
        __syncthreads();
    }
    if (RoleC) {
        // the last block to finish checks the hubs
        __syncthreads();  // every thread has read s_win
        if (threadIdx.x == 0) {
            __threadfence();
            s_win = atomicAdd(&ctl->dist_done, 1ull);
        }
        __syncthreads();
        if (s_win != gridDim.x - 1) return;
        __threadfence();
        hub_rows(0, 1, [&](int64_t e) {
            if ((int64_t)__ldcg(A.cnt + e) != __ldg(A.off + e + 1) - __ldg(A.off + e) - __ldg(A.cA + e) - __ldg(A.cB + e))
                atomicMax(A.status, (int)TDT_ERR_CAPACITY);
        });
    }
}

template <int M>
static int launch_walk(WalkArgs A, WalkCtl* ctl, cudaStream_t st) {
    DeviceInfo di;
    int rc = device_info(&di);
    if (rc) return rc;
    int wc = 0, hc = 0;
    support_caps(&wc, &hc);
    A.warp_cap = wc > 0 && wc < kLightCap ? wc : kLightCap;
    A.light_in = A.ne < kLightInEdges ? kLightInSmall : kLightInLarge;
    A.row_cap = hc > 0 && hc < kRowCap ? hc : kRowCap;
    auto kern = walk_kernel<M>;
    TDT_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kWkSmem));
    TDT_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, 100));
    int per_sm = 0;
    TDT_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kWkBlock, kWkSmem));
    if (per_sm < 1) per_sm = 1;
    const int64_t warps = (int64_t)di.sms * per_sm * kWkWarps;
    int64_t lb = A.nv / (warps * 4);  // at least four grabs a warp, so no warp is left with a long batch
    lb = lb < 1 ? 1 : (lb > kWarp ? kWarp : lb);
    kern<<<di.sms * per_sm, kWkBlock, kWkSmem, st>>>(A, ctl, (int)lb);
    TDT_LAUNCH_CHECK("walk");
    return TDT_OK;
}

static WalkArgs walk_args(const int64_t* rp, const int32_t* cols, const int64_t* cp, const int32_t* in_src,
                          const int32_t* in_eid, int64_t nv, int64_t ne, int32_t* cA, int32_t* cB, int32_t* cC,
                          const void* units, const int* gate, int* status) {
    WalkArgs A{};
    A.rp = rp;
    A.cols = cols;
    A.cp = cp;
    A.in_src = in_src;
    A.in_eid = in_eid;
    A.nv = nv;
    A.ne = ne;
    A.cA = cA;
    A.cB = cB;
    A.cC = cC;
    A.units = reinterpret_cast<const int2*>(units);
    A.gate = gate;
    A.status = status;
    return A;
}

// Plan and count walk: role counts of every edge and, when sbase (else null)
// needs no more than stage_slots, the role-A entries in their staging slots,
// which end at stage_end; *stage_skip receives the choice.  cA, cB, cC and ctl
// are zeroed by the caller.  units: 16 E bytes of scratch that stays as
// the list walk's plan; runA: int32[E] and longs: uint32[E] scratch; ctl: 256
// bytes.
int launch_walk_count(const int64_t* rp, const int32_t* cols, const int64_t* cp, const int32_t* in_src,
                      const int32_t* in_eid, int64_t nv, int64_t ne, int32_t* cA, int32_t* cB, int32_t* cC,
                      const int64_t* sbase, int2* stage_end, unsigned long long stage_slots, int* stage_skip,
                      int32_t* runA, void* units, void* longs, void* ctl, int* status, cudaStream_t st) {
    if (nv <= 0) return TDT_OK;
    DeviceInfo di;
    int rc = device_info(&di);
    if (rc) return rc;
    int wc = 0, hc = 0;
    support_caps(&wc, &hc);
    const int warp_cap = wc > 0 && wc < kLightCap ? wc : kLightCap;
    walk_plan_kernel<<<grid_for(nv, 256, di.sms, 8), 256, 0, st>>>(rp, cp, nv, warp_cap,
                                                                  ne < kLightInEdges ? kLightInSmall : kLightInLarge,
                                                                  reinterpret_cast<int2*>(units), hub_list(units, ne), sbase, stage_slots, stage_skip,
                                                                  reinterpret_cast<WalkCtl*>(ctl), status);
    TDT_LAUNCH_CHECK("walk_plan");
    WalkArgs A = walk_args(rp, cols, cp, in_src, in_eid, nv, ne, cA, cB, cC, units, status, status);
    A.sbase = sbase;
    A.out = stage_end;
    A.stage_skip = stage_skip;
    A.runA = runA;
    A.longs = reinterpret_cast<uint32_t*>(longs);
    return launch_walk<kWalkCount>(A, reinterpret_cast<WalkCtl*>(ctl), st);
}

// Role-A entries at their final places (off), after launch_walk_count with the
// same plan (skipped on the device when *gate != 0).
int launch_walk_list(const int64_t* rp, const int32_t* cols, const int64_t* cp, const int32_t* in_src,
                     const int32_t* in_eid, int64_t nv, int64_t ne, const int64_t* off, int32_t* cA, int2* lists,
                     int32_t* runA, void* units, void* longs, void* ctl, const int* gate, int* status,
                     cudaStream_t st) {
    if (nv <= 0) return TDT_OK;
    WalkArgs A = walk_args(rp, cols, cp, in_src, in_eid, nv, ne, cA, nullptr, nullptr, units, gate, status);
    A.off = off;
    A.out = lists;
    A.runA = runA;
    A.longs = reinterpret_cast<uint32_t*>(longs);
    return launch_walk<kWalkList>(A, reinterpret_cast<WalkCtl*>(ctl), st);
}

// Roles B and C of every list (and role A from the staging slots when
// *stage_skip == 0), skipped on the device when *gate != 0.  cnt:
// uint32[E], zeroed by the caller; units: the walk's plan.
int launch_distribute(const int64_t* rp, const int32_t* cols, const int32_t* rows, const int64_t* cp,
                      const int32_t* in_eid, int64_t nv, int64_t ne, const int64_t* off, const int32_t* cA,
                      const int32_t* cB, const int64_t* sbase, const int2* stage_end, const int* stage_skip,
                      int2* lists, uint32_t* cnt, void* units, void* ctl, const int* gate, int* status,
                      cudaStream_t st) {
    if (nv <= 0 || ne <= 0) return TDT_OK;
    DeviceInfo di;
    int rc = device_info(&di);
    if (rc) return rc;
    DistArgs A{rp, cols, rows, cp, in_eid, nv, ne, off, cA, cB, sbase, stage_end, stage_skip, lists,
               cnt, hub_list(units, ne), status, gate};
    for (int role = 0; role < 2; role++) {
        auto kern = role ? distribute_kernel<true> : distribute_kernel<false>;
        TDT_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kDsSmem));
        TDT_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, 100));
        int per_sm = 0;
        TDT_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kDsBlock, kDsSmem));
        if (per_sm < 1) per_sm = 1;
        kern<<<di.sms * per_sm, kDsBlock, kDsSmem, st>>>(A, reinterpret_cast<WalkCtl*>(ctl));
        TDT_LAUNCH_CHECK("distribute");
    }
    return TDT_OK;
}

}  // namespace tdt
