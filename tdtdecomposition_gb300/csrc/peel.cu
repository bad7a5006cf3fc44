// Device-resident truss decomposition and k-truss search.
//
// Replaces the `--cuda` flow's Python peel loop (singlegpu_truss.py:67-158:
// ~12 torch launches and ~6 host syncs per sub-round, each O(E)) by ONE
// persistent cooperative kernel that runs every sub-round and level on the
// device, separated by a bounded grid barrier.
//
// Per sub-round r at level l, F_r = edges peeled in r (rnd[e] == r):
//   * every e in F_r enumerates its triangles from the endpoint x of lower
//     degree: the candidates are x's out- and in-neighbours w; the third edge
//     between w and the other endpoint y is found by binary search in the
//     sorted out-list of min(w, y) (ids are degree ranks, so that list is
//     short);
//   * a triangle (e, f, g) whose edges were all alive at the start of r is
//     destroyed; f and g outside F_r lose one support each; when f (or g) is
//     also in F_r only the member with the smaller index decrements the third
//     edge; when all three are in F_r nothing is decremented;
//   * an edge whose support drops from l+1 to l joins F_{r+1}.
// When F_{r+1} is empty, the level advances to the minimum support of the
// alive edges and F_{r+1} = alive edges with that support.
// This yields exactly the reference's sub-round sets (singlegpu_truss.py:
// 99-152 with sub_AllAffectedSupport_tilenot, kernel.cu:492-547): each
// non-peeled edge loses one support per destroyed triangle, and an edge
// joins the next sub-round exactly when its support reaches <= l; so
// truss[e] = level + 2 and the reference's e_truss order (sub-rounds in
// order, ascending edge index within a sub-round) are reproduced exactly.
//
// Work in a sub-round is a flat candidate space: each queued edge owns
// deg(x) consecutive candidate slots (reserved with one packed 64-bit atomic
// per warp: item count in the high bits, candidate count in the low bits, so
// item order equals slot order), and every lane of the grid takes one slot
// per step.  Hub edges therefore spread over all SMs instead of one thread.
// With per-edge triangle lists (listed mode) a slot is one list entry: the
// two partner edges, whose states come from 4-bit round codes held in L2.
#include "common.cuh"
#include "sort.cuh"

namespace tdt {

#ifndef TDT_PEEL_BLOCK
#define TDT_PEEL_BLOCK 512
#endif
constexpr int kPeelBlock = TDT_PEEL_BLOCK;
constexpr int kPeelWarps = kPeelBlock / kWarp;
constexpr int kItemBits = 28;
constexpr int kCandBits = 36;
constexpr unsigned long long kCandMask = (1ull << kCandBits) - 1ull;
// Wall-clock budget of one persistent peel launch; past it the run stops with
// TDT_ERR_TIMEOUT instead of holding the GPU.
constexpr uint64_t kPeelDeadlineNs = 120ull * 1000ull * 1000ull * 1000ull;

struct PeelCtl {
    GridCtl g;
    // round r's counters live at r & 3: round r reads slot r, appends to r+1,
    // turns round r-1's edges dead, and the top of round r clears r+2
    unsigned long long q[4];      // packed (items << kCandBits | candidates) per round slot
    unsigned long long fe[4];     // frontier edges per round slot (queued or not)
    unsigned long long cnt[3];     // survivors written by level change t, at t % 3
    unsigned long long pfe[3];     // edges queued by level-change pass k, at k % 3
    int mgt[3];                    // minimum support found by level-change pass k, at k % 3
    int dmin[2];                   // minimum decrement result above the level during level L_t, at t & 1
    long long passes;              // level-change passes run (diagnostic)
    int listed;                   // 1: per-edge triangle lists were built (they fit the workspace)
    int list_skip;                // gate of the listing kernels (no lists)
    int stage_skip;               // the walk only counts
    int compact_skip;             // the role-A entries are not taken from the staging slots
    int rewalk_skip;              // gate of the list walk
    long long rounds;
    long long triangles;
    unsigned long long alive;
    // block 0's time (ns) in candidate processing, grid-barrier waits after
    // processing, and level transitions; diagnostic only
    unsigned long long t_proc, t_wait, t_trans, t_total;
    unsigned long long grab[4];    // slot cursor of search-mode sub-round r, at r & 3
    unsigned done;                 // blocks of a counting last kernel that finished
};

// How the peel finds an edge's triangles: in its list, by search in the graph's
// adjacency, or by search in an adjacency that is compacted as edges die.
enum PeelMode { kListed = 0, kSearch = 1, kCompact = 2 };
// The compacted adjacency: still the graph's own; compacted, with items queued
// before that; compacted.
enum CompactState { kWhole = 0, kStale = 1, kFresh = 2 };

struct PeelArgs {
    const int64_t* rp;
    const int32_t* cols;
    const int32_t* rows;
    const int64_t* cp;
    int32_t* in_src;
    int32_t* in_eid;
    int32_t* live;        // support of each edge, decremented as its triangles are destroyed
    int32_t* rnd;         // sub-round that peeled each edge (-1: alive)
    int32_t* round_level;
    // queue of round r in buffer r % 3: round r reads r, appends r+1, and the
    // items of round r-1 stay intact for the codes turned dead during round r
    int4* qi[3];
    long long* qb[3];
    int32_t* alive[2];    // compacted alive-edge lists (level transitions)
    // round r at r & 1: the item that holds slot 32 j, for j < kSlotIdx
    int32_t* sidx[2];
    // compacted adjacency (see compact_rows): row u's out-edges at rp[u] of
    // out_col / out_eid, its in-edges at cp[u] of in_src / in_eid, as many as its
    // lengths say
    int32_t* out_col;
    int32_t* out_eid;
    int32_t* out_len;
    int32_t* in_len;
    // round code of edge e in the 4 bits at (e & 7) * 4 of word e >> 3 (the
    // listed peel's partner-state check; see code_round)
    unsigned* code;
    const int64_t* off;   // listed mode: list offsets int64[E+1]
    const int2* lists;    // listed mode: partner edge pairs
    int64_t V, E, round_cap;
    int32_t mode;         // 0: full decomposition, 1: fixed-level peel (k-truss search)
    int32_t fixed_level;
    unsigned long long deadline_ns;  // wall-clock budget of the launch
    unsigned long long fixed_item_cap, fixed_cand_cap;  // k-truss collection batch limits
    long long dyn_min_slots;      // search mode: sub-rounds of at least this many slots take dynamic ranges
    int search_next;      // a search kernel follows the one that may find no lists
    PeelCtl* ctl;
};

__device__ __forceinline__ void set_status(PeelCtl* c, int s) {
    atomicMax(&c->g.status, s);
    grid_abort(&c->g);
}

// Round-boundary barrier of the persistent loop: arrivals counted against an
// epoch that every thread keeps (no returned value on the arrival), and the
// next sub-round's counters fetched by the waiting thread and handed to the
// block through shared memory, so no warp pays a load for them.
struct RoundBar {
    unsigned long long target;   // arrivals that complete the next barrier
    unsigned long long q, fe;    // counters of the round asked for (fe after a level change: edges it queued)
};

struct RoundShared {
    unsigned long long q, fe;
    int ok;
    int dmin;                    // smallest decrement result of the block's sub-round
    // level changes: edges alive, the alive list's length and which of the two it is (-1: every edge id)
    long long alive, nlist;
    int list;
};

__device__ __forceinline__ void red_release_add(unsigned long long* p, unsigned long long v) {
    asm volatile("red.release.gpu.global.add.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// Barrier over all blocks; next: the round whose counters are wanted.  dmin:
// where the block's smallest decrement result goes (reset for the next
// sub-round).  A wait of more than limit_ns sets TDT_ERR_TIMEOUT and aborts the
// run.  False when the run is being aborted.
__device__ __forceinline__ bool round_barrier(PeelCtl* ctl, RoundBar& B, RoundShared* S, int next, int* dmin,
                                              uint64_t limit_ns = kBarrierTimeoutNs) {
    __syncthreads();
    if (threadIdx.x == 0) {
        int ok = 1;
        if (S->dmin != INT32_MAX) {
            atomicMin(dmin, S->dmin);
            S->dmin = INT32_MAX;
        }
        red_release_add(&ctl->g.arrive, 1ull);
        const uint64_t t0 = globaltimer_ns();
        unsigned spins = 0;
        for (;;) {
            const unsigned long long v = ld_acquire_u64(&ctl->g.arrive);
            if (v & kGridAbortBit) {
                ok = 0;
                break;
            }
            if (v >= B.target) break;
            if ((++spins & 31u) == 0) {
                if (globaltimer_ns() - t0 > limit_ns) {
                    atomicMax(&ctl->g.status, (int)TDT_ERR_TIMEOUT);
                    grid_abort(&ctl->g);
                    ok = 0;
                    break;
                }
                if (spins > 4096) __nanosleep(200);
            }
        }
        S->q = __ldcg(&ctl->q[next & 3]);
        S->fe = __ldcg(&ctl->fe[next & 3]);
        S->ok = ok;
    }
    __syncthreads();
    B.target += gridDim.x;
    B.q = S->q;
    B.fe = S->fe;
    return S->ok != 0;
}

__device__ __forceinline__ unsigned long long ld_cg_u64(const unsigned long long* p) {
    return __ldcg(p);
}

// Round codes: 4 bits per edge, 32 MB at 64 M edges, so they stay in L2.
// 0xF: never marked (alive); 0-3: marked for sub-round y, stored as y & 3;
// bit 3 set: peeled and done.  A code is set once, when its edge is marked
// (0xF -> y & 3, one atomicAnd), and turned dead during sub-round y + 1
// (atomicOr 0x8 over the items of round y).  An edge marked without
// an item (no triangle left to enumerate) is dead at once: each of its
// triangles is already destroyed by a partner peeled before it.  Hence, in
// sub-round r (a grid barrier after every sub-round), a code reads 0xF
// alive, r & 3 peeling in r, (r + 1) & 3 marked for r + 1, and anything else
// peeled before r (an edge of r - 1 may still carry (r + 3) & 3).
constexpr unsigned kCodeAlive = 0xFu, kCodeDead = 0x8u;

__device__ __forceinline__ void code_mark(unsigned* code, int32_t e, unsigned c) {
    atomicAnd(code + (e >> 3), ~((kCodeAlive ^ c) << ((unsigned)(e & 7) * 4u)));
}

// The sub-round stamp of edge e read from its code word in sub-round r: -1
// alive, r or r + 1, or -2 for peeled before r.
__device__ __forceinline__ int32_t code_round(unsigned word, int32_t e, int r) {
    const unsigned c = (word >> ((unsigned)(e & 7) * 4u)) & 15u;
    if (c == kCodeAlive) return -1;
    if (c == ((unsigned)r & 3u)) return r;
    if (c == ((unsigned)(r + 1) & 3u)) return r + 1;
    return -2;
}

// Queue item of edge e (listed: e's list offset and length; search: the
// lower-degree endpoint x, the other endpoint y, x's out-degree dxo and the
// candidate count dx).  Returns false when e has nothing to enumerate.
template <int Mode>
__device__ __forceinline__ bool make_item(const PeelArgs& A, bool want, int32_t cur_sup, int32_t e, int4& it,
                                          long long& dx) {
    it = make_int4(e, 0, 0, 0);
    dx = 0;
    if (!want || cur_sup <= 0) return false;
    if (Mode == kListed) {
        // the edge's original triangles; the item carries the list offset
        const long long o = __ldg(A.off + e);
        dx = __ldg(A.off + e + 1) - o;
        it.y = (int32_t)(unsigned)(o & 0xffffffffll);
        it.z = (int32_t)(o >> 32);
        return dx > 0;
    }
    const int32_t u = __ldg(A.rows + e), v = __ldg(A.cols + e);
    if (Mode == kCompact) {
        const int32_t uo = __ldcg(A.out_len + u), vo = __ldcg(A.out_len + v);
        const int32_t du = uo + __ldcg(A.in_len + u), dv = vo + __ldcg(A.in_len + v);
        it.y = du <= dv ? u : v;
        it.z = du <= dv ? v : u;
        it.w = du <= dv ? uo : vo;
        dx = du <= dv ? du : dv;
        return dx > 1;
    }
    const long long duo = __ldg(A.rp + u + 1) - __ldg(A.rp + u);
    const long long du = duo + __ldg(A.cp + u + 1) - __ldg(A.cp + u);
    const long long dvo = __ldg(A.rp + v + 1) - __ldg(A.rp + v);
    const long long dv = dvo + __ldg(A.cp + v + 1) - __ldg(A.cp + v);
    if (du <= dv) { it.y = u; it.z = v; dx = du; it.w = (int32_t)duo; }
    else { it.y = v; it.z = u; dx = dv; it.w = (int32_t)dvo; }
    return dx > 1;
}

// 32-slot windows covered by the slot index.
constexpr int kSlotIdx = 32768;
// A listed sub-round takes the short chain up to this many windows a warp
// (peel at R-MAT scale 16 / 18 / 20: 7.52 / 14.04 / 34.55 ms with one, 7.38 /
// 13.79 / 33.95 with four, the same with six).
constexpr int kLeanWindows = 4;
// A search sub-round, whose slots cost from one load to twenty, takes its
// windows strided over the warps up to this many a warp: neighbouring slots,
// which cost alike, spread out (Chung-Lu, 1 M vertices: 120 ms of peel with one
// range a warp, 104 ms).
constexpr int kLeanSearch = 8;

// Records item idx, slots [c, c + dx), in the slot index of its round.
__device__ __forceinline__ void index_item(int32_t* sidx, long long idx, long long c, long long dx) {
    for (long long j = (c + kWarp - 1) / kWarp; j < kSlotIdx && j * kWarp < c + dx; j++) sidx[j] = (int32_t)idx;
}

// Reserve n items and tot candidate slots of the round in `slot` (lane 0's
// atomic, broadcast); sets TDT_ERR_CAPACITY past the queue limits.
__device__ __forceinline__ unsigned long long reserve_items(const PeelArgs& A, int slot, int n, long long tot) {
    unsigned long long old = 0;
    if (lane_id() == 0) {
        old = atomicAdd(&A.ctl->q[slot], ((unsigned long long)n << kCandBits) + (unsigned long long)tot);
        const unsigned long long it0 = old >> kCandBits, c0 = old & kCandMask;
        if (it0 + n >= (1ull << kItemBits) || c0 + tot >= (1ull << kCandBits) || (long long)(it0 + n) > A.E)
            set_status(A.ctl, TDT_ERR_CAPACITY);
    }
    return __shfl_sync(kFull, old, 0);
}

// Appends of the listed sub-rounds and of the level changes are staged per
// warp in shared memory (edge ids only, 256 bytes a warp, so the carveout
// leaves L1 its room) and queued in batches: one queue atomic (and one
// frontier-count atomic) per flush instead of two per warp step that marks an
// edge, which keeps the reservation's round trip and the contention on the
// round's counters out of most steps.  The items are built at the flush.  The
// queue order of items changes nothing: a sub-round is a set.
#ifndef TDT_APPEND_BUF
#define TDT_APPEND_BUF 64
#endif
constexpr int kAppBuf = TDT_APPEND_BUF;  // entries per warp; a flush leaves room for one 64-edge append
static_assert(kAppBuf >= 64 && kAppBuf % 32 == 0, "append buffer");

struct AppendBuf {
    int32_t* e;                  // this warp's staged edges (shared memory)
    int n;                       // staged edges (warp-uniform)
    unsigned long long nfront;   // edges marked since the last flush (warp-uniform)
};

// Queue the staged edges: their items are built here (kAppBuf / 32 per lane),
// reserved with one atomic and written.
template <int Mode>
__device__ __forceinline__ void append_flush(const PeelArgs& A, int slot, int buf, AppendBuf& B,
                                             unsigned long long* nfront) {
    const unsigned lane = lane_id();
    __syncwarp();
    if (B.nfront) {
        if (lane == 0) atomicAdd(nfront, B.nfront);
        B.nfront = 0;
    }
    if (B.n > 0) {
        constexpr int kPer = kAppBuf / kWarp;
        int4 it[kPer];
        long long dx[kPer];
        bool q[kPer];
        int nq = 0;
        long long sum = 0;
#pragma unroll
        for (int k = 0; k < kPer; k++) {
            const int i = (int)lane * kPer + k;
            q[k] = i < B.n && make_item<Mode>(A, true, 1, B.e[i], it[k], dx[k]);
            if (q[k]) {
                nq++;
                sum += dx[k];
            }
        }
        const int nincl = warp_incl_scan(nq);
        const int ntot = __shfl_sync(kFull, nincl, 31);
        const long long cincl = warp_incl_scan(sum);
        const long long ctot = __shfl_sync(kFull, cincl, 31);
        if (ntot > 0) {
            const unsigned long long old = reserve_items(A, slot, ntot, ctot);
            long long idx = (long long)(old >> kCandBits) + nincl - nq;
            long long cc = (long long)(old & kCandMask) + cincl - sum;
#pragma unroll
            for (int k = 0; k < kPer; k++) {
                if (q[k]) {
                    if (idx < A.E) {
                        A.qi[buf][idx] = it[k];
                        A.qb[buf][idx] = cc;
                        index_item(A.sidx[slot & 1], idx, cc, dx[k]);
                    }
                    idx++;
                    cc += dx[k];
                }
            }
        }
        B.n = 0;
    }
    __syncwarp();
}

// The same as a call (the level-change passes: several call sites, rare flushes).
template <int Mode>
__device__ __noinline__ void append_flush_call(const PeelArgs& A, int slot, int buf, AppendBuf& B,
                                               unsigned long long* nfront) {
    append_flush<Mode>(A, slot, buf, B, nfront);
}

// Stage up to two edges per lane (f, g of one triangle) for the round in
// `slot`; cur_sup (the level, warp-uniform) <= 0 queues no item.
template <int Mode>
__device__ __forceinline__ void warp_append2_staged(const PeelArgs& A, int slot, int buf, bool wf, int32_t f,
                                                    bool wg, int32_t g, int32_t cur_sup, AppendBuf& B,
                                                    unsigned long long* nfront) {
    const unsigned mf = __ballot_sync(kFull, wf), mg = __ballot_sync(kFull, wg);
    if ((mf | mg) == 0) return;
    B.nfront += (unsigned long long)(__popc(mf) + __popc(mg));
    if (cur_sup <= 0) return;
    const int nq = (wf ? 1 : 0) + (wg ? 1 : 0);
    const int nincl = warp_incl_scan(nq);
    const int ntot = __shfl_sync(kFull, nincl, 31);
    if (B.n + ntot > kAppBuf) append_flush<Mode>(A, slot, buf, B, nfront);
    int p = B.n + nincl - nq;
    if (wf) B.e[p++] = f;
    if (wg) B.e[p] = g;
    B.n += ntot;
}

// Queue up to two edges per lane directly, with one reservation per warp step
// (the search-mode sub-rounds: their steps are long and append rarely, and the
// staging state would stay live across the binary searches).
template <int Mode>
__device__ __forceinline__ void warp_append2_direct(const PeelArgs& A, int slot, int buf, bool wf, int32_t f,
                                                    bool wg, int32_t g, int32_t cur_sup,
                                                    unsigned long long* nfront) {
    const unsigned lane = lane_id();
    const unsigned mf = __ballot_sync(kFull, wf), mg = __ballot_sync(kFull, wg);
    if ((mf | mg) == 0) return;
    if (lane == 0) atomicAdd(nfront, (unsigned long long)(__popc(mf) + __popc(mg)));
    int4 itf, itg;
    long long dxf, dxg;
    const bool qf = make_item<Mode>(A, wf, cur_sup, f, itf, dxf);
    const bool qg = make_item<Mode>(A, wg, cur_sup, g, itg, dxg);
    const int nq = (qf ? 1 : 0) + (qg ? 1 : 0);
    if (__ballot_sync(kFull, nq > 0) == 0) return;
    const long long c = (qf ? dxf : 0) + (qg ? dxg : 0);
    const int nincl = warp_incl_scan(nq);
    const long long cincl = warp_incl_scan(c);
    const int ntot = __shfl_sync(kFull, nincl, 31);
    const long long ctot = __shfl_sync(kFull, cincl, 31);
    const unsigned long long old = reserve_items(A, slot, ntot, ctot);
    long long idx = (long long)(old >> kCandBits) + nincl - nq;
    long long cc = (long long)(old & kCandMask) + cincl - c;
    if (qf) {
        if (idx < A.E) {
            A.qi[buf][idx] = itf;
            A.qb[buf][idx] = cc;
            index_item(A.sidx[slot & 1], idx, cc, dxf);
        }
        idx++;
        cc += dxf;
    }
    if (qg && idx < A.E) {
        A.qi[buf][idx] = itg;
        A.qb[buf][idx] = cc;
        index_item(A.sidx[slot & 1], idx, cc, dxg);
    }
}

// Stage the edges flagged by `want` (one per lane) for the round in `slot`.
// cur_sup is the edge's support at marking time (0 => no alive triangle).
template <int Search>
__device__ __forceinline__ void warp_append_staged(const PeelArgs& A, bool listed, int slot, int buf, bool want,
                                                   int32_t e, int32_t cur_sup, AppendBuf& B,
                                                   unsigned long long* nfront) {
    const unsigned mf = __ballot_sync(kFull, want);
    if (mf == 0) return;
    B.nfront += (unsigned long long)__popc(mf);
    const bool st = want && cur_sup > 0;
    const unsigned m = __ballot_sync(kFull, st);
    if (m == 0) return;
    const int ntot = __popc(m);
    if (B.n + ntot > kAppBuf) {
        if (listed) append_flush_call<kListed>(A, slot, buf, B, nfront);
        else append_flush_call<Search>(A, slot, buf, B, nfront);
    }
    if (st) B.e[B.n + __popc(m & lanemask_lt())] = e;
    B.n += ntot;
}

// Level changes (decomposition mode).  Level change t starts level L_t =
// min support over the alive edges and queues F = alive edges with support
// L_t.  The alive edges lie among the entries of a list, every edge id at
// first, rewritten from one array into the other when enough of it has died.
//
// One streaming pass usually suffices: a lower bound g of L_t is known before
// the pass (0 at t = 0; afterwards the minimum support above L_{t-1} seen at
// change t-1, lowered by every decrement result above L_{t-1} during level
// L_{t-1}).  The pass may rewrite the list, queues the alive edges with
// support == g, and takes the minimum support above g.  If
// anything was queued, L_t = g.  Otherwise L_t = that minimum, and one more
// pass over the list queues its frontier (3 of 307 level changes
// at R-MAT scale 22; a side list of the supports just above g, written by
// every first pass for that case, cost the level changes 3 ms there).  Every
// pass k ends with a grid barrier and writes its minimum and queued count to
// slot k % 3 of mgt / pfe; the block-0 thread that clears slot (k+1) % 3 at
// the start of pass k clears a slot that every block finished reading before
// the barrier of pass k-1.

// Fold a per-lane minimum into *dst: one atomic per warp, skipped when *dst
// is already no larger (a plain read keeps ten thousand warps from
// serialising on one address).
__device__ __forceinline__ void fold_min(int* dst, int32_t v) {
    v = warp_min(v);
    if (lane_id() == 0 && v != INT32_MAX && v < *(volatile int*)dst) atomicMin(dst, v);
}

__device__ __forceinline__ void pass_min(const PeelArgs& A, int np, int32_t v) { fold_min(&A.ctl->mgt[np % 3], v); }

// A level change rewrites the alive list only when a kListSlack-th of it has
// died; until then its dead entries cost a code word each, and until the first
// rewrite the list is every edge id and is not read at all.  Level changes are
// bound by these passes on large graphs: rewritten every time 19.1 ms at R-MAT
// scale 22 (307 level changes), 5.7 at 20, 0.99 at 16; now 14.2, 4.7 and 0.83 (a third
// instead of an eighth: 14.7, 4.7, 0.81).
constexpr int kListSlack = 8;

// Level-change passes stream the alive list in steps of kStep x 32 entries per
// warp: the gathers of a step are in flight together and the step reserves its
// output ranges with one atomic each.
#ifndef TDT_DYN_CHUNK
#define TDT_DYN_CHUNK 256
#endif
#ifndef TDT_DYN_MIN_LOG2
#define TDT_DYN_MIN_LOG2 20
#endif
constexpr long long kDynChunk = TDT_DYN_CHUNK;  // 0: static ranges in search mode too
constexpr int kDynMinLog2 = TDT_DYN_MIN_LOG2;
static_assert(kDynChunk % 64 == 0, "dynamic ranges are whole 64-slot steps");
// An edge already marked for sub-round r+1 (support <= l) is not decremented
// again: its support no longer decides anything (it is peeled next sub-round,
// and its truss number is the level).
#ifndef TDT_SKIP_MARKED
#define TDT_SKIP_MARKED 1
#endif
constexpr bool kSkipMarked = TDT_SKIP_MARKED != 0;
#ifndef TDT_PEEL_STEP
#define TDT_PEEL_STEP 8
#endif
constexpr int kStep = TDT_PEEL_STEP;

__device__ __forceinline__ void pass_start(const PeelArgs& A, int np) {
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        A.ctl->mgt[(np + 1) % 3] = INT32_MAX;
        A.ctl->pfe[(np + 1) % 3] = 0;
        A.ctl->passes++;
    }
}

// Search: the mode when the peel is not listed.
template <int Search>
__device__ __forceinline__ bool level_transition(const PeelArgs& A, bool listed, int r_next, int t, int& np,
                                              int32_t* l_out, int32_t* app_e, RoundBar& RB, RoundShared* RS) {
    const unsigned lane = lane_id();
    const long long gw = (long long)blockIdx.x * kPeelWarps + threadIdx.x / kWarp;
    const long long nw = (long long)gridDim.x * kPeelWarps;
    const bool first = t == 0;
    const int p = RS->list;
    const int32_t* cur = p < 0 ? nullptr : A.alive[p];
    int32_t* nxt = A.alive[p < 0 ? 0 : p ^ 1];
    const long long ncur = RS->nlist;
    const bool write = RS->alive < ncur - ncur / kListSlack;
    int32_t g = 0;
    if (!first) {
        const int32_t a = *(volatile int*)&A.ctl->mgt[(np + 2) % 3];
        const int32_t b = *(volatile int*)&A.ctl->dmin[(t + 1) & 1];
        g = a < b ? a : b;
    }
    const int slot = r_next & 3, buf = r_next % 3;
    AppendBuf B{app_e + (threadIdx.x / kWarp) * kAppBuf, 0, 0ull};
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        A.ctl->cnt[(t + 1) % 3] = 0;
        A.ctl->dmin[t & 1] = INT32_MAX;
    }
    pass_start(A, np);
    // pass 1: compact, queue support == g, minimum above g.  Blocks take
    // tiles of kPeelWarps x kStep x 32 entries; each tile reserves its
    // survivor range with one atomic.
    {
        __shared__ int s_tk[kPeelWarps];
        __shared__ unsigned long long s_base;
        constexpr long long kTile = (long long)kPeelWarps * kStep * kWarp;
        const int wib = threadIdx.x / kWarp;
        int32_t mloc = INT32_MAX;
        unsigned long long* ocnt = &A.ctl->cnt[t % 3];
        const unsigned lt = lanemask_lt();
        for (long long tb = (long long)blockIdx.x * kTile; tb < ncur; tb += (long long)gridDim.x * kTile) {
            const long long base = tb + (long long)wib * (kStep * kWarp);
            int32_t e[kStep], sv[kStep];
            bool keep[kStep];
#pragma unroll
            for (int u = 0; u < kStep; u++) {
                const long long i = base + u * kWarp + lane;
                e[u] = 0;
                if (i < ncur) e[u] = cur ? __ldcg(cur + i) : (int32_t)i;
            }
#pragma unroll
            for (int u = 0; u < kStep; u++) {
                const long long i = base + u * kWarp + lane;
                keep[u] = false;
                sv[u] = 0;
                if (i < ncur) {
                    // alive = never marked (its round code, in L2); the
                    // support is a 4-byte gather
                    const unsigned cw = __ldcg(A.code + (e[u] >> 3));
                    sv[u] = __ldcg(A.live + e[u]);
                    keep[u] = ((cw >> ((unsigned)(e[u] & 7) * 4u)) & 15u) == kCodeAlive;
                }
            }
            unsigned km[kStep];
            int nk = 0;
#pragma unroll
            for (int u = 0; u < kStep; u++) {
                km[u] = __ballot_sync(kFull, keep[u]);
                nk += __popc(km[u]);
                if (keep[u] && sv[u] > g) mloc = sv[u] < mloc ? sv[u] : mloc;
            }
            if (write) {
                if (lane == 0) s_tk[wib] = nk;
                __syncthreads();
            }
            if (write && wib == 0) {
                const int a = lane < kPeelWarps ? s_tk[lane] : 0;
                const int ai = warp_incl_scan(a);
                if (lane == kPeelWarps - 1) s_base = ai ? atomicAdd(ocnt, (unsigned long long)ai) : 0ull;
                if (lane < kPeelWarps) s_tk[lane] = ai - a;
            }
            unsigned long long ok = 0;
            if (write) {
                __syncthreads();
                ok = s_base + (unsigned long long)s_tk[wib];
            }
#pragma unroll
            for (int u = 0; u < kStep; u++) {
                if (write) {
                    if (keep[u]) nxt[ok + __popc(km[u] & lt)] = e[u];
                    ok += __popc(km[u]);
                }
                const bool want = keep[u] && sv[u] == g;
                if (want) {
                    A.rnd[e[u]] = r_next;
                    code_mark(A.code, e[u], sv[u] > 0 ? ((unsigned)r_next & 3u) : kCodeDead);
                }
                warp_append_staged<Search>(A, listed, slot, buf, want, e[u], sv[u], B, &A.ctl->pfe[np % 3]);
            }
            if (write) __syncthreads();  // s_tk / s_base are reused by the next tile
        }
        if (listed) append_flush_call<kListed>(A, slot, buf, B, &A.ctl->pfe[np % 3]);
        else append_flush_call<Search>(A, slot, buf, B, &A.ctl->pfe[np % 3]);
        pass_min(A, np, mloc);
    }
    np++;
    if (!round_barrier(A.ctl, RB, RS, r_next, &A.ctl->dmin[t & 1])) return false;
    RB.fe = ld_cg_u64(&A.ctl->pfe[(np + 2) % 3]);
    if (write && threadIdx.x == 0) {  // every thread has read the state, and reads it again after other barriers
        RS->list = p < 0 ? 0 : p ^ 1;
        RS->nlist = (long long)__ldcg(&A.ctl->cnt[t % 3]);
    }
    if (RB.fe > 0) {
        *l_out = g;
        return true;
    }
    const int32_t m = *(volatile int*)&A.ctl->mgt[(np + 2) % 3];
    if (m == INT32_MAX) return false;  // no edge is alive
    *l_out = m;
    pass_start(A, np);
    int32_t mloc = INT32_MAX;
    {
        // pass 2: one more pass over the list
        const long long n2 = write ? (long long)__ldcg(&A.ctl->cnt[t % 3]) : ncur;
        for (long long base = gw * kWarp; base < n2; base += nw * kWarp) {
            const long long i = base + lane;
            int32_t e = 0, sv = INT32_MAX;
            if (i < n2) {
                e = write ? __ldcg(nxt + i) : cur ? __ldcg(cur + i) : (int32_t)i;
                const unsigned cw = __ldcg(A.code + (e >> 3));
                if (((cw >> ((unsigned)(e & 7) * 4u)) & 15u) == kCodeAlive) sv = __ldcg(A.live + e);
            }
            const bool want = sv == m;  // m < INT32_MAX
            if (!want && sv > m) mloc = sv < mloc ? sv : mloc;
            if (want) {
                A.rnd[e] = r_next;
                code_mark(A.code, e, sv > 0 ? ((unsigned)r_next & 3u) : kCodeDead);
            }
            warp_append_staged<Search>(A, listed, slot, buf, want, e, sv, B, &A.ctl->pfe[np % 3]);
        }
    }
    if (listed) append_flush_call<kListed>(A, slot, buf, B, &A.ctl->pfe[np % 3]);
    else append_flush_call<Search>(A, slot, buf, B, &A.ctl->pfe[np % 3]);
    pass_min(A, np, mloc);
    np++;
    if (!round_barrier(A.ctl, RB, RS, r_next, &A.ctl->dmin[t & 1])) return false;
    RB.fe = ld_cg_u64(&A.ctl->pfe[(np + 2) % 3]);
    return true;
}

// k-truss search (fixed level l): the frontier is every alive edge with
// support <= l, collected in batches.  A collection pass queues such edges
// while the round's queue stays under fixed_item_cap items and fixed_cand_cap
// candidate slots (by default far below the packed counter's limits, which
// leaves room for warps that read the count before others added to it);
// edges left out stay alive and are taken by the next pass, which runs
// whenever a sub-round queues nothing.  The k-truss does not depend on how the
// peel is split into rounds, so the batches change no result; they keep the
// rounds of graphs whose low-support edges outnumber the queue within it.
constexpr unsigned long long kFixedItemCap = 1ull << 27;
constexpr unsigned long long kFixedCandCap = 1ull << 35;

template <int Search>
__device__ __forceinline__ void warp_append_capped(const PeelArgs& A, bool listed, int slot, int buf, bool want,
                                                   int32_t e,
                                                   int32_t s, int r_next, unsigned long long* nfront) {
    const unsigned lane = lane_id();
    if (__ballot_sync(kFull, want) == 0) return;
    int4 it;
    long long dx;
    const bool q = listed ? make_item<kListed>(A, want, s, e, it, dx) : make_item<Search>(A, want, s, e, it, dx);
    const unsigned m = __ballot_sync(kFull, q);
    const long long c = q ? dx : 0;
    const long long incl = warp_incl_scan(c);
    const long long tot = __shfl_sync(kFull, incl, 31);
    const int n = __popc(m);
    int ok = 1;
    unsigned long long old = 0;
    if (lane == 0 && n > 0) {
        const unsigned long long cur = ld_cg_u64(&A.ctl->q[slot]);
        // a batch always takes something (an empty queue accepts any warp)
        if (cur != 0 && ((cur >> kCandBits) + (unsigned long long)n > A.fixed_item_cap ||
                         (cur & kCandMask) + (unsigned long long)tot > A.fixed_cand_cap)) {
            ok = 0;
        } else {
            old = atomicAdd(&A.ctl->q[slot], ((unsigned long long)n << kCandBits) + (unsigned long long)tot);
            const unsigned long long it0 = old >> kCandBits, c0 = old & kCandMask;
            if (it0 + n >= (1ull << kItemBits) || c0 + tot >= (1ull << kCandBits) || (long long)(it0 + n) > A.E)
                set_status(A.ctl, TDT_ERR_CAPACITY);
        }
    }
    ok = __shfl_sync(kFull, ok, 0);
    old = __shfl_sync(kFull, old, 0);
    // edges without candidates use no queue space and are always taken
    const bool acc = want && (!q || ok);
    if (acc) {
        A.rnd[e] = r_next;
        code_mark(A.code, e, q ? ((unsigned)r_next & 3u) : kCodeDead);
    }
    const unsigned ma = __ballot_sync(kFull, acc);
    if (lane == 0 && ma) atomicAdd(nfront, (unsigned long long)__popc(ma));
    if (q && ok) {
        const long long idx = (long long)(old >> kCandBits) + __popc(m & lanemask_lt());
        if (idx < A.E) {
            A.qi[buf][idx] = it;
            A.qb[buf][idx] = (long long)(old & kCandMask) + incl - c;
            index_item(A.sidx[slot & 1], idx, (long long)(old & kCandMask) + incl - c, dx);
        }
    }
}

// One collection pass for sub-round r_next; true when it took an edge.
template <int Search>
__device__ bool fixed_collect(const PeelArgs& A, bool listed, int32_t l, int r_next, int& np, RoundBar& RB,
                              RoundShared* RS) {
    const unsigned lane = lane_id();
    const int64_t nthreads = (int64_t)gridDim.x * blockDim.x;
    const int slot = r_next & 3, buf = r_next % 3;
    pass_start(A, np);
    for (int64_t base = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) & ~31ll; base < A.E;
         base += nthreads) {
        const int64_t e = base + lane;
        bool want = false;
        int32_t s = 0;
        if (e < A.E) {
            const unsigned cw = __ldcg(A.code + (e >> 3));
            s = __ldcg(A.live + e);
            want = ((cw >> ((unsigned)(e & 7) * 4u)) & 15u) == kCodeAlive && s <= l;
        }
        warp_append_capped<Search>(A, listed, slot, buf, want, (int32_t)e, s, r_next, &A.ctl->pfe[np % 3]);
    }
    np++;
    if (!round_barrier(A.ctl, RB, RS, r_next, &A.ctl->dmin[0])) return false;
    RB.fe = ld_cg_u64(&A.ctl->pfe[(np + 2) % 3]);
    return RB.fe > 0;
}

// Item windows: slot cb lies in item i0 (first slot base0); items i0+1.. start
// at strictly increasing slots, all > cb, so at most 31 start inside
// (cb, cb+32).  One OR-reduction gives every lane the item of slot cb+lane.
struct Window {
    int k;              // this lane's item is i0 + k
    long long base_l;   // first slot of that item
    long long i0n;      // item of slot cb+32
    long long base0n;   // its first slot
    long long nsn;      // first slot of item i0n + 1 (-1: not among the loaded starts)
    bool starts_next;   // item i0n starts at cb+32 (no lane of this window holds it)
};

__device__ __forceinline__ Window locate(const long long* __restrict__ qb, long long N, long long i0,
                                         long long base0, long long cb, unsigned le) {
    const unsigned lane = lane_id();
    const long long B = (i0 + 1 + lane < N) ? __ldcg(qb + i0 + 1 + lane) : LLONG_MAX;
    const unsigned bit = (B - cb < kWarp) ? (1u << (unsigned)(B - cb)) : 0u;
    const unsigned mk = __reduce_or_sync(kFull, bit);
    Window w;
    w.k = __popc(mk & le);
    const long long Bk = __shfl_sync(kFull, B, (w.k + 31) & 31);
    w.base_l = w.k == 0 ? base0 : Bk;
    const int nb = __popc(mk);
    const long long Bn = __shfl_sync(kFull, B, nb);
    const long long Bl = __shfl_sync(kFull, B, (nb + 31) & 31);
    const long long B2 = __shfl_sync(kFull, B, (nb + 1) & 31);
    w.starts_next = Bn == cb + kWarp;
    if (w.starts_next) {
        w.i0n = i0 + nb + 1;
        w.base0n = Bn;
        w.nsn = nb + 1 < kWarp ? B2 : -1;
    } else {
        w.i0n = i0 + nb;
        w.base0n = nb > 0 ? Bl : base0;
        w.nsn = nb < kWarp ? Bn : -1;
    }
    return w;
}

// The items of one window [cb, cb + 32) of a warp's range: this lane's item
// record and first slot.  The warp keeps its current item i0 (holding slot
// cb, or ending just before it when item i0 + 1 starts at cb; locate handles
// both), that item's first slot, the first slot of the next item (nst, -1 when
// unknown) and the item's record (rec, valid when rv): a window that lies
// wholly in item i0 -- most windows, since most slots belong to long lists --
// needs no load at all; otherwise one locate step and one record load per
// lane, which also refresh the state.
__device__ __forceinline__ void window_items(const long long* __restrict__ qb, const int4* __restrict__ qi,
                                             long long N, long long cb, bool valid, unsigned le, long long& i0,
                                             long long& base0, long long& nst, int4& rec, bool& rv, int4& it,
                                             long long& base_l) {
    if (nst >= cb + kWarp) {
        if (!rv) {
            rec = __ldcg(qi + i0);
            rv = true;
        }
        it = rec;
        base_l = base0;
        return;
    }
    const Window w = locate(qb, N, i0, base0, cb, le);
    it = make_int4(0, 0, 0, 0);
    if (valid) it = __ldcg(qi + i0 + w.k);
    base_l = w.base_l;
    // lane 31 holds item i0n unless that item starts at cb + 32 (or lane 31
    // lies past the range)
    const bool v31 = (__ballot_sync(kFull, valid) >> 31) != 0u;
    rec.x = __shfl_sync(kFull, it.x, 31);
    rec.y = __shfl_sync(kFull, it.y, 31);
    rec.z = __shfl_sync(kFull, it.z, 31);
    rec.w = __shfl_sync(kFull, it.w, 31);
    rv = v31 && !w.starts_next;
    i0 = w.i0n;
    base0 = w.base0n;
    nst = w.nsn;
}

// Search mode: the other two edges (f, g) of slot tl[h] of item it[h] and their
// sub-round stamps, for the kWin windows of a step; tr[h] (in: the slot exists)
// turns false when the slot is no triangle or needs no decrement from here.
// A slot is a chain of loads, most of them the binary search for the third
// edge, so the windows go through each stage together: their searches run in
// step, kWin loads in flight instead of one.
#ifndef TDT_PEEL_WIN
#define TDT_PEEL_WIN 2
#endif
constexpr int kWin = TDT_PEEL_WIN;  // 32-slot windows per peel step

template <int Mode>
__device__ __forceinline__ void search_slots(const PeelArgs& A, const int4 (&it)[kWin], const int (&tl)[kWin], int r,
                                             int cst, bool (&tr)[kWin], int32_t (&f)[kWin], int32_t (&g)[kWin],
                                             int32_t (&rf)[kWin], int32_t (&rg)[kWin]) {
    // before the first compaction the rows are the graph's own
    const bool whole = Mode != kCompact || cst == kWhole;
    const int32_t* out_col = whole ? A.cols : A.out_col;
    int32_t w[kWin];
#pragma unroll
    for (int h = 0; h < kWin; h++) {
        w[h] = f[h] = g[h] = 0;
        rf[h] = rg[h] = -2;
        if (Mode == kCompact && tr[h]) {
            const bool o = tl[h] < it[h].w;
            const int i = o ? tl[h] : tl[h] - it[h].w;
            // an item queued before the last compaction has the lengths of then
            tr[h] = cst != kStale || i < __ldcg((o ? A.out_len : A.in_len) + it[h].y);
            if (tr[h]) {
                const int64_t k = __ldg((o ? A.rp : A.cp) + it[h].y) + i;
                w[h] = __ldcg((o ? out_col : A.in_src) + k);
                f[h] = o && whole ? (int32_t)k : __ldcg((o ? A.out_eid : A.in_eid) + k);
                tr[h] = w[h] != it[h].z;
            }
        } else if (tr[h]) {
            if (tl[h] < it[h].w) {
                f[h] = (int32_t)(__ldg(A.rp + it[h].y) + tl[h]);
                w[h] = __ldg(A.cols + f[h]);
            } else {
                const int64_t kk = __ldg(A.cp + it[h].y) + (tl[h] - it[h].w);
                w[h] = __ldg(A.in_src + kk);
                f[h] = __ldg(A.in_eid + kk);
            }
            tr[h] = w[h] != it[h].z;
        }
    }
    unsigned x[kWin];
#pragma unroll
    for (int h = 0; h < kWin; h++) x[h] = tr[h] ? __ldcg(A.code + (f[h] >> 3)) : 0u;
    int64_t b[kWin];
    int n[kWin];
    int32_t key[kWin];
    bool any = false;
#pragma unroll
    for (int h = 0; h < kWin; h++) {
        b[h] = 0;
        n[h] = 0;
        key[h] = 0;
        // no search when (x,w) was peeled before this round, or peels in it
        // too with the smaller index: then the other edge of the triangle is
        // decremented from (x,w)'s own slot, not from this one
        rf[h] = tr[h] ? code_round(x[h], f[h], r) : -2;
        tr[h] = tr[h] && rf[h] != -2 && !(rf[h] == r && it[h].x > f[h]);
        if (tr[h]) {
            const int32_t y = it[h].z, src = w[h] < y ? w[h] : y;
            key[h] = w[h] < y ? y : w[h];
            b[h] = __ldg(A.rp + src);
            n[h] = Mode == kCompact ? __ldcg(A.out_len + src) : (int)(__ldg(A.rp + src + 1) - b[h]);
        }
        tr[h] = n[h] > 0;
        any |= n[h] > 1;
    }
    // the last entry <= key of each list, in step
    while (any) {
        any = false;
        int32_t c[kWin];
#pragma unroll
        for (int h = 0; h < kWin; h++) {
            c[h] = INT32_MAX;
            if (n[h] > 1) c[h] = Mode == kCompact ? out_col[b[h] + (n[h] >> 1)] : __ldg(A.cols + b[h] + (n[h] >> 1));
        }
#pragma unroll
        for (int h = 0; h < kWin; h++) {
            const int half = n[h] >> 1;
            if (c[h] <= key[h]) b[h] += half;
            n[h] -= half;
            any |= n[h] > 1;
        }
    }
#pragma unroll
    for (int h = 0; h < kWin; h++) {
        g[h] = (int32_t)b[h];
        if (Mode == kCompact) {
            if (tr[h] && !whole) g[h] = A.out_eid[b[h]];
            tr[h] = tr[h] && out_col[b[h]] == key[h];
        } else {
            tr[h] = tr[h] && __ldg(A.cols + b[h]) == key[h];
        }
    }
#pragma unroll
    for (int h = 0; h < kWin; h++) {
        x[h] = tr[h] ? __ldcg(A.code + (g[h] >> 3)) : 0u;
    }
#pragma unroll
    for (int h = 0; h < kWin; h++) rg[h] = tr[h] ? code_round(x[h], g[h], r) : -2;
}

// The decrements of one peel step: the four edges and the supports before
// their decrements (INT32_MIN: no decrement).  An edge whose support fell to
// l is marked for sub-round r+1 and queued; a larger result lowers the bound
// dm of the next level.
struct Pending {
    int32_t e[2 * kWin];
    int32_t o[2 * kWin];
};

template <int Mode>
__device__ __forceinline__ void settle(const PeelArgs& A, const Pending& P, int r, int32_t l, int nslot, int nbuf,
                                       AppendBuf& B, int32_t& dm) {
    constexpr bool Listed = Mode == kListed;
    bool w[2 * kWin];
    // queued with an item when the level is above 0 (an edge without
    // triangles never appears in a list, so its code is never read)
    const unsigned cm = l > 0 ? ((unsigned)(r + 1) & 3u) : kCodeDead;
#pragma unroll
    for (int j = 0; j < 2 * kWin; j++) {
        w[j] = P.o[j] == l + 1;
        if (P.o[j] > l + 1) dm = P.o[j] - 1 < dm ? P.o[j] - 1 : dm;
        if (w[j]) {
            A.rnd[P.e[j]] = r + 1;
            code_mark(A.code, P.e[j], cm);
        }
    }
#pragma unroll
    for (int h = 0; h < kWin; h++) {
        if (Listed)
            warp_append2_staged<Mode>(A, nslot, nbuf, w[2 * h], P.e[2 * h], w[2 * h + 1], P.e[2 * h + 1], l, B,
                                        &A.ctl->fe[nslot]);
        else
            warp_append2_direct<Mode>(A, nslot, nbuf, w[2 * h], P.e[2 * h], w[2 * h + 1], P.e[2 * h + 1], l,
                                        &A.ctl->fe[nslot]);
    }
}

// A listed sub-round of a few windows a warp: a chain of dependent loads with
// nothing to hide it (300 cycles each in L2, 500 for an atomic's result), so
// the chain is kept short.  The slot index gives the window's first item, the
// records and first slots of the 32 items from it on come together, and a lane
// takes its record by shuffles: slot index, items, list entry, round codes,
// decrement, instead of counters, item search (a load per factor of 32), item,
// window starts, records, list entry, codes, decrement.  With the counters
// handed over by the barrier, peel of R-MAT scale 12 / 16 / 20 / 22: 2.58 /
// 9.70 / 40.3 / 116.6 -> 1.72 / 7.32 / 33.6 / 104.2 ms.
template <int Mode>
__device__ __forceinline__ void lean_round(const PeelArgs& A, int r, int32_t l, int N, int T, int gwarp, int nwarps,
                                           int32_t* ebuf, int* s_dmin, int cst) {
    constexpr bool Listed = Mode == kListed;
    if (gwarp * kWarp >= T) return;
    const unsigned lane = lane_id();
    const unsigned le = lanemask_lt() | (1u << lane);
    const int buf = r % 3, nslot = (r + 1) & 3, nbuf = (r + 1) % 3;
    const unsigned cm = l > 0 ? ((unsigned)(r + 1) & 3u) : kCodeDead;
    int32_t dm = INT32_MAX;
    AppendBuf B{ebuf, 0, 0ull};
    constexpr int kL = Listed ? 1 : kWin;  // windows in flight
    for (int cb0 = gwarp * kWarp; cb0 < T; cb0 += kL * nwarps * kWarp) {
        int i0[kL];
#pragma unroll
        for (int h = 0; h < kL; h++) {
            const int cb = cb0 + h * nwarps * kWarp;
            i0[h] = cb < T ? __ldcg(A.sidx[r & 1] + (cb >> 5)) : N;
        }
        int4 it[kL];
        int S[kL];  // first slot of item i0 + lane
#pragma unroll
        for (int h = 0; h < kL; h++) {
            it[h] = make_int4(0, 0, 0, 0);
            S[h] = INT32_MAX;
            if (i0[h] + (int)lane < N) {
                it[h] = __ldcg(A.qi[buf] + i0[h] + lane);
                S[h] = (int)__ldcg(A.qb[buf] + i0[h] + lane);
            }
        }
        int tl[kL];
        bool v[kL];
#pragma unroll
        for (int h = 0; h < kL; h++) {
            const int cb = cb0 + h * nwarps * kWarp;
            const unsigned d = (unsigned)(S[h] - cb);
            const unsigned mk = __reduce_or_sync(kFull, lane > 0 && d < (unsigned)kWarp ? 1u << d : 0u);
            const int k = __popc(mk & le);
            v[h] = cb + (int)lane < T;
            tl[h] = cb + (int)lane - __shfl_sync(kFull, S[h], k);
            it[h].x = __shfl_sync(kFull, it[h].x, k);
            it[h].y = __shfl_sync(kFull, it[h].y, k);
            it[h].z = __shfl_sync(kFull, it[h].z, k);
            if (!Listed) it[h].w = __shfl_sync(kFull, it[h].w, k);
        }
        int32_t f[kL], g[kL], rf[kL], rg[kL];
        if constexpr (Listed) {
            int2 fg = make_int2(0, 0);
            if (v[0]) fg = __ldg(A.lists + ((long long)(unsigned)it[0].y | ((long long)it[0].z << 32)) + tl[0]);
            f[0] = fg.x;
            g[0] = fg.y;
            unsigned xf = 0, xg = 0;
            if (v[0]) {
                xf = __ldcg(A.code + (fg.x >> 3));
                xg = __ldcg(A.code + (fg.y >> 3));
            }
            rf[0] = v[0] ? code_round(xf, fg.x, r) : -2;
            rg[0] = v[0] ? code_round(xg, fg.y, r) : -2;
        } else {
            search_slots<Mode>(A, it, tl, r, cst, v, f, g, rf, rg);
#pragma unroll
            for (int h = 0; h < kL; h++)
                if (!v[h]) rf[h] = -2;
        }
        // the ownership rules of process_round
        int32_t of[kL], og[kL];
#pragma unroll
        for (int h = 0; h < kL; h++) {
            const bool on = rf[h] != -2 && rg[h] != -2;
            const bool cf = rf[h] == r, cg = rg[h] == r;
            of[h] = og[h] = INT32_MIN;
            if (on && !cf && (!cg || it[h].x < g[h]) && (!kSkipMarked || rf[h] != r + 1))
                of[h] = atomicSub(A.live + f[h], 1);
            if (on && !cg && (!cf || it[h].x < f[h]) && (!kSkipMarked || rg[h] != r + 1))
                og[h] = atomicSub(A.live + g[h], 1);
        }
#pragma unroll
        for (int h = 0; h < kL; h++) {
            if (of[h] > l + 1 && of[h] - 1 < dm) dm = of[h] - 1;
            if (og[h] > l + 1 && og[h] - 1 < dm) dm = og[h] - 1;
            const bool wf = of[h] == l + 1, wg = og[h] == l + 1;
            if (wf) {
                A.rnd[f[h]] = r + 1;
                code_mark(A.code, f[h], cm);
            }
            if (wg) {
                A.rnd[g[h]] = r + 1;
                code_mark(A.code, g[h], cm);
            }
            warp_append2_staged<Mode>(A, nslot, nbuf, wf, f[h], wg, g[h], l, B, &A.ctl->fe[nslot]);
        }
    }
    dm = warp_min(dm);
    if (lane == 0 && dm != INT32_MAX) atomicMin(s_dmin, dm);
    append_flush<Mode>(A, nslot, nbuf, B, &A.ctl->fe[nslot]);
}

// One sub-round: warps gwarp = 0..nwarps-1 share the candidate slots of round r.
// The smallest decrement result above l is folded into *dmin (the lower bound
// of the next level).  Each step covers two 32-slot windows whose loads and
// decrements are in flight together.  Inlined into the persistent loop (with
// the level changes): the kernel arguments are a __grid_constant__ parameter,
// so no call passes a local copy of them, and no call frame is saved around
// every sub-round.
template <int Mode>
__device__ __forceinline__ void process_round(const PeelArgs& A, int r, int32_t l, unsigned long long packed,
                                              long long nprev, long long gwarp, long long nwarps, int* s_dmin,
                                              int32_t* app_e, int cst) {
    constexpr bool Listed = Mode == kListed;
    const unsigned lane = lane_id();
    const unsigned le = lanemask_lt() | (1u << lane);
    int32_t dm = INT32_MAX;
    const int slot = r & 3, buf = r % 3;
    const int nslot = (r + 1) & 3, nbuf = (r + 1) % 3;
    const int wib = threadIdx.x / kWarp;
    AppendBuf B{app_e + wib * kAppBuf, 0, 0ull};
    const long long N = (long long)(packed >> kCandBits);
    const long long T = (long long)(packed & kCandMask);
    const long long* __restrict__ qb = A.qb[buf];
    const int4* __restrict__ qi = A.qi[buf];
    // the edges of round r-1 are dead from this round on: their round codes
    // turn dead (needed by round r+2, where (r-1) & 3 would read "marked for
    // the next round")
    if (r > 0) {
        const int4* __restrict__ qp = A.qi[(r - 1) % 3];
        for (long long i = gwarp * kWarp + lane; i < nprev; i += nwarps * kWarp) {
            const int32_t e = __ldcg(&qp[i].x);
            atomicOr(A.code + (e >> 3), kCodeDead << ((unsigned)(e & 7) * 4u));
        }
    }
    if (T <= nwarps * kWarp * (Listed ? kLeanWindows : kLeanSearch) && T <= (long long)kSlotIdx * kWarp) {
        lean_round<Mode>(A, r, l, (int)N, (int)T, (int)gwarp, (int)nwarps, app_e + wib * kAppBuf, s_dmin, cst);
        return;
    }
    // listed mode: each warp owns a contiguous range of candidate slots (a
    // multiple of 64).  Search mode with many slots: warps take ranges of
    // kDynChunk slots from a shared cursor (the binary search of a slot costs
    // from one load to twenty, so equal ranges finish far apart).
    const bool dyn = !Listed && kDynChunk > 0 && T >= A.dyn_min_slots;
    constexpr long long kStepSlots = (long long)kWin * kWarp;
    const long long per_warp = (((T + nwarps - 1) / nwarps) + kStepSlots - 1) / kStepSlots * kStepSlots;
    long long cb0 = gwarp * per_warp;
    long long cb1 = cb0 + per_warp < T ? cb0 + per_warp : T;
    if (!dyn && cb0 >= cb1) return;
    Pending P;
#pragma unroll
    for (int j = 0; j < 2 * kWin; j++) {
        P.e[j] = 0;
        P.o[j] = INT32_MIN;
    }
    for (;;) {
    if (dyn) {
        unsigned long long c = 0;
        if (lane == 0) c = atomicAdd(&A.ctl->grab[slot], (unsigned long long)kDynChunk);
        cb0 = (long long)__shfl_sync(kFull, c, 0);
        if (cb0 >= T) break;
        cb1 = cb0 + kDynChunk < T ? cb0 + kDynChunk : T;
    }
    // item of slot cb0 = last i with qb[i] <= cb0: a 32-way search, each step
    // one load per lane (log32 N dependent loads instead of log2 N)
    long long i0 = 0;
    {
        long long lo = 0, hi = N;  // answer in [lo, hi)
        while (hi - lo > 1) {
            const long long step = (hi - lo + kWarp - 1) / kWarp;
            const long long p = lo + (long long)lane * step;
            const bool le_ = p < hi && __ldcg(qb + p) <= cb0;
            const unsigned m = __ballot_sync(kFull, le_);
            const int j = 31 - __clz(m);  // qb[lo] <= cb0 always holds, so m != 0
            lo += (long long)j * step;
            hi = lo + step < hi ? lo + step : hi;
        }
        i0 = lo;
    }
    long long base0 = __ldcg(qb + i0);
    long long nst = i0 + 1 < N ? __ldcg(qb + i0 + 1) : LLONG_MAX;
    int4 rec = __ldcg(qi + i0);
    bool rv = true;
    for (long long cb = cb0; cb < cb1; cb += kStepSlots) {
        int4 it[kWin];
        long long bl[kWin];
        bool v[kWin];
#pragma unroll
        for (int h = 0; h < kWin; h++) {
            const long long cbh = cb + h * kWarp;
            it[h] = make_int4(0, 0, 0, 0);
            bl[h] = 0;
            v[h] = cbh + lane < cb1;
            if (cbh < cb1) window_items(qb, qi, N, cbh, v[h], le, i0, base0, nst, rec, rv, it[h], bl[h]);
        }
        int32_t f[kWin], g[kWin], rf[kWin], rg[kWin];
        bool tr[kWin];
        if (Listed) {
            // list entry, then the partners' round codes (L2): dead, alive,
            // peeling now, marked
            unsigned x[kWin], y[kWin];
#pragma unroll
            for (int h = 0; h < kWin; h++) {
                f[h] = g[h] = 0;
                tr[h] = false;
                if (v[h]) {
                    const long long lo = (long long)(unsigned)it[h].y | ((long long)it[h].z << 32);
                    const int2 fg = __ldg(A.lists + lo + (cb + h * kWarp + lane - bl[h]));
                    f[h] = fg.x;
                    g[h] = fg.y;
                    tr[h] = true;
                }
            }
#pragma unroll
            for (int h = 0; h < kWin; h++) rf[h] = rg[h] = -2;
#pragma unroll
            for (int h = 0; h < kWin; h++) {
                x[h] = y[h] = 0;
                if (tr[h]) {
                    x[h] = __ldcg(A.code + (f[h] >> 3));
                    y[h] = __ldcg(A.code + (g[h] >> 3));
                }
            }
            // the previous step's decrement results, while these loads are in flight
            settle<Mode>(A, P, r, l, nslot, nbuf, B, dm);
#pragma unroll
            for (int h = 0; h < kWin; h++) {
                if (tr[h]) {
                    rf[h] = code_round(x[h], f[h], r);
                    rg[h] = code_round(y[h], g[h], r);
                }
            }
        } else {
            int tl[kWin];
#pragma unroll
            for (int h = 0; h < kWin; h++) {
                tl[h] = (int)(cb + h * kWarp + lane - bl[h]);
                tr[h] = v[h];
            }
            search_slots<Mode>(A, it, tl, r, cst, tr, f, g, rf, rg);
            settle<Mode>(A, P, r, l, nslot, nbuf, B, dm);
        }
        // a triangle is alive when both other edges are alive or peel in r or r+1;
        // which of f, g this lane decrements: the ownership rules above
        bool df[kWin], dg[kWin];
#pragma unroll
        for (int h = 0; h < kWin; h++) {
            df[h] = dg[h] = false;
            if (tr[h] && (rf[h] == -1 || rf[h] >= r) && (rg[h] == -1 || rg[h] >= r)) {
                const bool ff = rf[h] == r, fg = rg[h] == r;
                df[h] = !ff && (!fg || it[h].x < g[h]) && (!kSkipMarked || rf[h] != r + 1);
                dg[h] = !fg && (!ff || it[h].x < f[h]) && (!kSkipMarked || rg[h] != r + 1);
            }
        }
        // issue all decrements; their results are used by the next step
#pragma unroll
        for (int h = 0; h < kWin; h++) {
            P.e[2 * h] = f[h];
            P.e[2 * h + 1] = g[h];
        }
#pragma unroll
        for (int h = 0; h < kWin; h++) {
            P.o[2 * h] = df[h] ? atomicSub(A.live + f[h], 1) : INT32_MIN;
            P.o[2 * h + 1] = dg[h] ? atomicSub(A.live + g[h], 1) : INT32_MIN;
        }
    }
    if (!dyn) break;
    }
    settle<Mode>(A, P, r, l, nslot, nbuf, B, dm);
    if (Listed) append_flush<Mode>(A, nslot, nbuf, B, &A.ctl->fe[nslot]);
    dm = warp_min(dm);
    if (lane == 0 && dm != INT32_MAX) atomicMin(s_dmin, dm);
}

// The search peel walks a peeled edge's neighbours, dead edges among them, and
// they cost it a round-code load each.  Its rows are therefore compacted (order
// and row starts kept, lengths shrunk; the first time into a copy, then in
// place) whenever the alive edges have halved: every compaction reads what the
// one before left, so all of them together read about twice the edges, and the
// slots of a Chung-Lu graph fall from 3.1 to 1.1 a list entry (host model, 60 K
// vertices).  Peel of one of 1 M vertices: 104 -> 69 ms, 3 ms of them in
// compactions (a quarter off instead of half: 72 ms).
__device__ __forceinline__ void compact_init(const PeelArgs& A) {
    const int64_t nth = (int64_t)gridDim.x * kPeelBlock, tid = (int64_t)blockIdx.x * kPeelBlock + threadIdx.x;
    for (int64_t u = tid; u < A.V; u += nth) {
        A.out_len[u] = (int32_t)(__ldg(A.rp + u + 1) - __ldg(A.rp + u));
        A.in_len[u] = (int32_t)(__ldg(A.cp + u + 1) - __ldg(A.cp + u));
    }
}

constexpr long long kCompactMin = 4096;  // alive edges at the last compaction below which there is no next one
constexpr int kCompactLong = 1024;  // rows longer than this are compacted by a block

// An edge stays until its sub-round is over: alive, or marked for sub-round r.
__device__ __forceinline__ bool compact_keep(const PeelArgs& A, int32_t e, int r) {
    const unsigned c = (__ldcg(A.code + (e >> 3)) >> ((unsigned)(e & 7) * 4u)) & 15u;
    return c == kCodeAlive || c == ((unsigned)r & 3u);
}

// One row's out- or in-edges by a warp or by the block, kCompactPer entries a
// thread at a time; returns the new length.
constexpr int kCompactPer = 4;

template <bool Out, bool Block>
__device__ __forceinline__ int compact_row(const PeelArgs& A, int64_t base, int len, int r, bool whole,
                                           int* s_warp) {
    const unsigned lane = lane_id();
    const int wib = threadIdx.x / kWarp;
    constexpr int kThr = Block ? kPeelBlock : kWarp;
    constexpr int kPer = Block ? kCompactPer : 1;
    const int tid = Block ? (int)threadIdx.x : (int)lane;
    int32_t* ids = (Out ? A.out_col : A.in_src) + base;
    int32_t* eids = (Out ? A.out_eid : A.in_eid) + base;
    int n = 0;
    for (int t = 0; t < len; t += kPer * kThr) {
        int2 x[kPer];
        bool keep[kPer];
        unsigned m[kPer];
#pragma unroll
        for (int j = 0; j < kPer; j++) {
            const int i = t + j * kThr + tid;
            x[j] = make_int2(0, -1);
            if (i < len) {
                if (Out && whole) x[j] = make_int2(__ldg(A.cols + base + i), (int32_t)(base + i));
                else x[j] = make_int2(__ldcg(ids + i), __ldcg(eids + i));
            }
        }
#pragma unroll
        for (int j = 0; j < kPer; j++) keep[j] = x[j].y >= 0 && compact_keep(A, x[j].y, r);
#pragma unroll
        for (int j = 0; j < kPer; j++) {
            m[j] = __ballot_sync(kFull, keep[j]);
            if (Block && lane == 0) s_warp[j * kPeelWarps + wib] = __popc(m[j]);
        }
        int all = __popc(m[0]), at = 0;
        if (Block) {
            __syncthreads();  // also: every entry of this tile has been read
            all = 0;
        } else {
            __syncwarp();  // the same: a vote orders no memory
        }
#pragma unroll
        for (int j = 0; j < kPer; j++) {
            if (Block) {
                at = all;
                for (int w = 0; w < kPeelWarps; w++) {
                    const int c = s_warp[j * kPeelWarps + w];
                    if (w < wib) at += c;
                    all += c;
                }
            }
            if (keep[j]) {
                const int to = n + at + __popc(m[j] & lanemask_lt());
                ids[to] = x[j].x;
                eids[to] = x[j].y;
            }
        }
        n += all;
        if (Block) __syncthreads();
        else __syncwarp();
    }
    return n;
}

// Drops the edges peeled before sub-round r from every row (a grid barrier
// follows).  A block takes kPeelBlock rows at a time, a thread reading the
// lengths of one: a warp compacts its 32 rows one after the other, then the
// block the long ones.  The rows of a block lie far apart in rank: the hubs are
// the top ranks, side by side.
__device__ __forceinline__ void compact_rows(const PeelArgs& A, int r, bool whole, int* s_warp, int32_t* s_rows) {
    __shared__ int s_n;
    const unsigned lane = lane_id();
    const int64_t stride = (A.V + kPeelBlock - 1) / kPeelBlock;
    for (int64_t b = blockIdx.x; b < stride; b += gridDim.x) {
        const int64_t u = b + threadIdx.x * stride;
        int lo = 0, li = 0;
        int64_t po = 0, pi = 0;
        if (u < A.V) {
            lo = __ldcg(A.out_len + u);
            li = __ldcg(A.in_len + u);
            po = __ldg(A.rp + u);
            pi = __ldg(A.cp + u);
        }
        if (threadIdx.x == 0) s_n = 0;
        __syncthreads();
        if (lo > kCompactLong || li > kCompactLong) s_rows[atomicAdd(&s_n, 1)] = (int32_t)threadIdx.x;
        unsigned m = __ballot_sync(kFull, lo > 0 && lo <= kCompactLong);
        while (m) {
            const int k = __ffs(m) - 1;
            m &= m - 1;
            const int n = compact_row<true, false>(A, __shfl_sync(kFull, po, k), __shfl_sync(kFull, lo, k), r, whole, nullptr);
            if ((int)lane == k) A.out_len[u] = n;
        }
        m = __ballot_sync(kFull, li > 0 && li <= kCompactLong);
        while (m) {
            const int k = __ffs(m) - 1;
            m &= m - 1;
            const int n = compact_row<false, false>(A, __shfl_sync(kFull, pi, k), __shfl_sync(kFull, li, k), r, whole, nullptr);
            if ((int)lane == k) A.in_len[u] = n;
        }
        __syncthreads();
        const int rows = s_n;
        for (int i = 0; i < rows; i++) {
            const int64_t v = b + s_rows[i] * stride;
            const int vo = __ldcg(A.out_len + v), vi = __ldcg(A.in_len + v);
            __syncthreads();
            // a length at or under the bound was settled by its warp
            if (vo > kCompactLong) {
                const int n = compact_row<true, true>(A, __ldg(A.rp + v), vo, r, whole, s_warp);
                if (threadIdx.x == 0) A.out_len[v] = n;
            }
            if (vi > kCompactLong) {
                const int n = compact_row<false, true>(A, __ldg(A.cp + v), vi, r, whole, s_warp);
                if (threadIdx.x == 0) A.in_len[v] = n;
            }
        }
        __syncthreads();
    }
}

#ifndef TDT_PEEL_MINB
#define TDT_PEEL_MINB 2
#endif
// A is a __grid_constant__ parameter: the helpers take it by reference and
// read its fields from the parameter bank instead of a local copy.
// kListed: the caller gave a list tail, and whether the lists fit is decided on
// the device (search otherwise).  Without a tail the search peels have kernels,
// and their registers, of their own (Chung-Lu, 1 M vertices, without
// compaction: 121 -> 104 ms).  A fixed level does not compact: at most levels its
// work is its first sub-rounds (k = 10 / 100 at R-MAT scale 20 6.7 / 40.0 ms, with
// compaction 7.0 / 41.7; k = 200 58.2 / 56.3, kmax 58.9 / 60.7; Chung-Lu, 1 M
// vertices, at kmax 33.9 / 32.1).
template <int Mode>
__global__ void __launch_bounds__(kPeelBlock, TDT_PEEL_MINB) peel_kernel(const __grid_constant__ PeelArgs A) {
    __shared__ int32_t s_app_e[kPeelWarps * kAppBuf];  // per-warp append staging
    __shared__ RoundShared s_round;
    __shared__ int s_warp[kCompactPer * kPeelWarps];
    const bool lists = *(volatile int*)&A.ctl->listed != 0;
    const bool listed = Mode == kListed && lists;
    if (Mode == kListed ? !lists && A.search_next : lists) return;
    constexpr int kOther = Mode == kCompact ? kCompact : kSearch;
    const int wib = threadIdx.x / kWarp;
    const int64_t gwarp = (int64_t)blockIdx.x * kPeelWarps + wib;
    const int64_t nwarps = (int64_t)gridDim.x * kPeelWarps;
    const bool master = blockIdx.x == 0 && threadIdx.x == 0;

    if (*(volatile int*)&A.ctl->g.status != 0) return;  // invalid input was detected
    const uint64_t t_start = globaltimer_ns();
    int r = 0;
    int32_t l = 0;
    int ntrans = 0, np = 0;
    bool ok;
    if (threadIdx.x == 0) {
        s_round.dmin = INT32_MAX;
        s_round.alive = s_round.nlist = A.E;
        s_round.list = -1;
    }
    __syncthreads();
    RoundBar RB{gridDim.x, 0ull, 0ull};
    long long nprev = 0;  // items of the sub-round before
    // compaction: edges alive now and at the last one
    long long alive = A.E, alive_c = A.E;
    int cst = kWhole;
    if constexpr (Mode == kCompact) {
        compact_init(A);
        if (!round_barrier(A.ctl, RB, &s_round, 0, &A.ctl->dmin[0])) return;
    }
    if (A.mode == 0) {
        ok = level_transition<kOther>(A, listed, 0, ntrans++, np, &l, s_app_e, RB, &s_round);
    } else {
        l = A.fixed_level;
        ok = fixed_collect<kOther>(A, listed, l, 0, np, RB, &s_round);
    }
    if (!ok) {
        if (master) A.ctl->rounds = 0;
        return;
    }
    alive -= (long long)RB.fe;
    if (threadIdx.x == 0) s_round.alive -= (long long)RB.fe;
    uint64_t t_mark = globaltimer_ns();
    for (;;) {
        if (master) {
            A.round_level[r] = l;
            A.ctl->q[(r + 2) & 3] = 0;
            A.ctl->fe[(r + 2) & 3] = 0;
            A.ctl->grab[(r + 2) & 3] = 0;
            if (globaltimer_ns() - t_start > A.deadline_ns) set_status(A.ctl, TDT_ERR_TIMEOUT);
        }
        if (listed) process_round<kListed>(A, r, l, RB.q, nprev, gwarp, nwarps, &s_round.dmin, s_app_e, kWhole);
        else process_round<kOther>(A, r, l, RB.q, nprev, gwarp, nwarps, &s_round.dmin, s_app_e, cst);
        if (cst == kStale) cst = kFresh;
        nprev = (long long)(RB.q >> kCandBits);
        if (nprev > A.E) nprev = A.E;
        __syncthreads();
        const uint64_t t_p = globaltimer_ns();
        // level L_t (t = ntrans - 1) folds its decrement results into dmin[t & 1]
        if (!round_barrier(A.ctl, RB, &s_round, r + 1, &A.ctl->dmin[(ntrans + 1) & 1])) return;
        const uint64_t t_b = globaltimer_ns();
        if (master) {
            A.ctl->t_proc += t_p - t_mark;
            A.ctl->t_wait += t_b - t_p;
        }
        if (r + 2 >= A.round_cap) {
            if (master) set_status(A.ctl, TDT_ERR_CAPACITY);
            return;
        }
        // fe[(r+1) & 3] is only written by sub-round r (level changes count
        // into pfe), and cleared again at the top of sub-round r+3
        if (RB.fe == 0) {
            if (A.mode != 0) {
                // k-truss search: the next batch of low-support edges, if any
                if (!fixed_collect<kOther>(A, listed, l, r + 1, np, RB, &s_round)) break;
                t_mark = globaltimer_ns();
                r++;
                alive -= (long long)RB.fe;
                continue;
            }
            int32_t nl;
            const bool more = level_transition<kOther>(A, listed, r + 1, ntrans++, np, &nl, s_app_e, RB, &s_round);
            if (master) A.ctl->t_trans += globaltimer_ns() - t_b;
            if (!more) break;
            l = nl;
        }
        if (threadIdx.x == 0) s_round.alive -= (long long)RB.fe;
        t_mark = globaltimer_ns();
        r++;
        if constexpr (Mode == kCompact) {
            alive -= (long long)RB.fe;
            if (2 * alive <= alive_c && alive_c >= kCompactMin) {
                compact_rows(A, r, cst == kWhole, s_warp, s_app_e);
                alive_c = alive;
                cst = kStale;
                if (!round_barrier(A.ctl, RB, &s_round, r, &A.ctl->dmin[(ntrans + 1) & 1])) return;
            }
        }
    }
    if (master) {
        A.ctl->rounds = r + 1;
        A.ctl->t_total = globaltimer_ns() - t_start;
    }
}

// ------------------------------------------------------------------ setup / output kernels
// Input validation, before any kernel indexes through the graph:
// row_ptr[0] == 0, row_ptr[V] == E, non-decreasing; rows[e] is the row that
// owns position e; u < v < V; columns strictly increasing within a row.
__device__ __forceinline__ int validate_edge(int32_t v, int32_t next, int64_t e, int64_t u, int64_t b, int64_t en,
                                             int64_t V) {
    if (u < 0 || u >= V || v >= V || u >= v) return TDT_ERR_NOT_ORIENTED;
    if (e < b || e >= en) return TDT_ERR_INVALID;
    return e + 1 < en && next <= v ? TDT_ERR_INVALID : TDT_OK;
}

// The column after edge e in a row that ends at en.
__device__ __forceinline__ int32_t next_col(const int32_t* __restrict__ cols, int64_t e, int64_t en) {
    return e + 1 < en ? cols[e + 1] : 0;
}

__global__ void validate_kernel(const int64_t* __restrict__ rp, const int32_t* __restrict__ rows,
                                const int32_t* __restrict__ cols, int64_t E, int64_t V, PeelCtl* ctl) {
    const int64_t tid = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int64_t nth = (int64_t)gridDim.x * blockDim.x;
    if (tid == 0 && (rp[0] != 0 || rp[V] != E)) atomicMax(&ctl->g.status, (int)TDT_ERR_INVALID);
    for (int64_t u = tid; u < V; u += nth)
        if (rp[u] > rp[u + 1]) atomicMax(&ctl->g.status, (int)TDT_ERR_INVALID);
    for (int64_t e = tid; e < E; e += nth) {
        const int32_t u = rows[e];
        const bool in = u >= 0 && u < V;
        const int64_t end = in ? rp[u + 1] : 0, en = end < E ? end : E;  // cols ends at E
        const int err = validate_edge(cols[e], next_col(cols, e, en), e, u, in ? rp[u] : 0, en, V);
        if (err) atomicMax(&ctl->g.status, err);
    }
}

// The same when the caller gave no rows: a warp per row writes them, inside
// [0, E) whatever row_ptr says.  Rows of more than kValLong edges wait in shared
// memory for the whole block, with kValUnroll edges a thread in flight: degree
// ranks have few of them, but a low hub's row in one warp is a chain of loads
// (a row of 2 M edges: 39 ms in a warp, 1.8 in a block).  Eight blocks per SM: the
// short rows wait for loads too (validation of scale 21 0.13 ms longer at six).
constexpr int kValBlock = 256;
constexpr int kValLong = 2048, kValList = 64, kValUnroll = 4;

__global__ void __launch_bounds__(kValBlock, 8) validate_rows_kernel(const int64_t* __restrict__ rp,
                                                                  int32_t* __restrict__ rows,
                                                                  const int32_t* __restrict__ cols, int64_t E,
                                                                  int64_t V, PeelCtl* ctl) {
    __shared__ int32_t s_long[kValList];
    __shared__ int s_n;
    const unsigned lane = lane_id();
    const int64_t tid = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    if (threadIdx.x == 0) s_n = 0;
    __syncthreads();
    if (tid == 0 && (rp[0] != 0 || rp[V] != E)) atomicMax(&ctl->g.status, (int)TDT_ERR_INVALID);
    for (int64_t u = tid >> 5; u < V; u += nw) {
        const int64_t b = rp[u], en = rp[u + 1];
        if (b > en || b < 0 || en > E) {
            atomicMax(&ctl->g.status, (int)TDT_ERR_INVALID);
            continue;
        }
        if (en - b > kValLong) {
            int at = 0;
            if (lane == 0) at = atomicAdd(&s_n, 1);
            at = __shfl_sync(kFull, at, 0);
            if (at < kValList) {
                if (lane == 0) s_long[at] = (int32_t)u;
                continue;
            }
        }
        for (int64_t e = b + lane; e < en; e += kWarp) {
            rows[e] = (int32_t)u;
            const int err = validate_edge(cols[e], next_col(cols, e, en), e, u, b, en, V);
            if (err) atomicMax(&ctl->g.status, err);
        }
    }
    __syncthreads();
    const int n = s_n < kValList ? s_n : kValList;
    for (int i = 0; i < n; i++) {
        const int64_t u = s_long[i], b = rp[u], en = rp[u + 1];
        for (int64_t e0 = b + threadIdx.x; e0 < en; e0 += kValUnroll * kValBlock) {
            int32_t v[kValUnroll], next[kValUnroll];
#pragma unroll
            for (int k = 0; k < kValUnroll; k++) {
                const int64_t e = e0 + k * kValBlock;
                v[k] = e < en ? cols[e] : 0;
                next[k] = next_col(cols, e, en);
            }
            int err = TDT_OK;
#pragma unroll
            for (int k = 0; k < kValUnroll; k++) {
                const int64_t e = e0 + k * kValBlock;
                if (e < en) {
                    rows[e] = (int32_t)u;
                    err = max(err, validate_edge(v[k], next[k], e, u, b, en, V));
                }
            }
            if (err) atomicMax(&ctl->g.status, err);
        }
    }
}

// In-adjacency.  Ids are degree ranks, so most heads are among the top ids and
// a hub's counter would take one atomic per in-edge, one after the other (7 to
// 9 ns each).  A block counts the heads of its edges among the top kCscHot ids
// in shared memory and adds each counter to the global one once; the fill then
// reserves a run of the in-list per (block, top id) and takes places in it from
// shared memory.  Both kernels at R-MAT scale 16 / 18 / 22: 145 us / 490 us /
// 4.1 ms with an atomic per edge, 39 us / 93 us / 2.0 ms.  The in-lists come out
// nearly in source order, and the walk that follows them fell from 1.10 to
// 0.51 ms at scale 18, from 8.4 to 6.8 ms at scale 21.
constexpr int kCscBlock = 512;
constexpr int kCscHot = 8192;
// Edges of a tile of the fill in a large graph: the places that the resident
// blocks write at one time stay within L2 (scale 22: 3.37 ms with one share a
// block, 2.85 with 65,536, 1.71 with 16,384, 1.66 with 4,096).
constexpr int kCscTile = 8192;
constexpr int kCscUnroll = 4;

// f(e, cols[e]) over edges [e0, e1) by the block.
template <class F>
__device__ __forceinline__ void csc_edges(const int32_t* __restrict__ cols, int64_t e0, int64_t e1, F&& f) {
    for (int64_t e = e0 + threadIdx.x; e < e1; e += kCscUnroll * kCscBlock) {
        int32_t v[kCscUnroll];
#pragma unroll
        for (int k = 0; k < kCscUnroll; k++) v[k] = e + k * kCscBlock < e1 ? __ldg(cols + e + k * kCscBlock) : -1;
#pragma unroll
        for (int k = 0; k < kCscUnroll; k++)
            if (v[k] >= 0) f(e + k * kCscBlock, v[k]);
    }
}

__global__ void __launch_bounds__(kCscBlock) indeg_kernel(const int32_t* __restrict__ cols, int64_t E, int64_t V,
                                                          int32_t* __restrict__ indeg, const PeelCtl* ctl) {
    __shared__ int32_t s_cnt[kCscHot];
    if (*(volatile const int*)&ctl->g.status != 0) return;
    const int32_t hot0 = V > kCscHot ? (int32_t)(V - kCscHot) : 0;
    const int hot = (int)(V - hot0);
    for (int i = threadIdx.x; i < hot; i += kCscBlock) s_cnt[i] = 0;
    __syncthreads();
    const int64_t per = (E + gridDim.x - 1) / gridDim.x, e0 = blockIdx.x * per;
    csc_edges(cols, e0, e0 + per < E ? e0 + per : E, [&](int64_t, int32_t v) {
        if (v >= hot0) atomicAdd(s_cnt + (v - hot0), 1);
        else atomicAdd(indeg + v, 1);
    });
    __syncthreads();
    for (int i = threadIdx.x; i < hot; i += kCscBlock)
        if (s_cnt[i]) atomicAdd(indeg + hot0 + i, s_cnt[i]);
}

// left: the in-degrees, counted down to zero as the in-lists fill from their ends.
__global__ void __launch_bounds__(kCscBlock) csc_fill_kernel(const int32_t* __restrict__ rows,
                                                             const int32_t* __restrict__ cols, int64_t E, int64_t V,
                                                             int64_t tile,
                                                             const int64_t* __restrict__ cp,
                                                             int32_t* __restrict__ left, int32_t* __restrict__ in_src,
                                                             int32_t* __restrict__ in_eid, const PeelCtl* ctl) {
    __shared__ int32_t s_cur[kCscHot];  // counts, then the next place of the block's run
    if (*(volatile const int*)&ctl->g.status != 0) return;
    const int32_t hot0 = V > kCscHot ? (int32_t)(V - kCscHot) : 0;
    const int hot = (int)(V - hot0);
    for (int64_t e0 = blockIdx.x * tile; e0 < E; e0 += gridDim.x * tile) {
        const int64_t e1 = e0 + tile < E ? e0 + tile : E;
        for (int i = threadIdx.x; i < hot; i += kCscBlock) s_cur[i] = 0;
        __syncthreads();
        csc_edges(cols, e0, e1, [&](int64_t, int32_t v) {
            if (v >= hot0) atomicAdd(s_cur + (v - hot0), 1);
        });
        __syncthreads();
        for (int i = threadIdx.x; i < hot; i += kCscBlock)
            if (s_cur[i])
                s_cur[i] = (int32_t)__ldg(cp + hot0 + i) + atomicSub(left + hot0 + i, s_cur[i]) - s_cur[i];
        __syncthreads();
        csc_edges(cols, e0, e1, [&](int64_t e, int32_t v) {
            const int32_t pos = v >= hot0 ? atomicAdd(s_cur + (v - hot0), 1)
                                          : (int32_t)__ldg(cp + v) + atomicSub(left + v, 1) - 1;
            in_src[pos] = __ldg(rows + e);
            in_eid[pos] = (int32_t)e;
        });
        __syncthreads();
    }
}

// sup = cA + cB + cC (the role counts of the walk) and the triangle total; for
// a peel also the edge state (live = sup, no sub-round, code alive).  A count
// (live null) ends here: sup is the caller's array or null, and the last block
// writes the stats.
__global__ void init_state_kernel(const int32_t* __restrict__ cA, const int32_t* __restrict__ cB,
                                  const int32_t* __restrict__ cC, int32_t* __restrict__ sup,
                                  int32_t* __restrict__ live, int32_t* __restrict__ rnd,
                                  unsigned* __restrict__ code, int64_t E, PeelCtl* ctl, int64_t* __restrict__ stats) {
    __shared__ long long s_part[32];
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        for (int i = 0; i < 3; i++) ctl->mgt[i] = INT32_MAX;
        ctl->dmin[0] = INT32_MAX;
        ctl->dmin[1] = INT32_MAX;
    }
    const int64_t tid = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, nth = (int64_t)gridDim.x * blockDim.x;
    long long acc = 0;
    for (int64_t e = tid; e < E; e += nth) {
        const int32_t s = cA[e] + cB[e] + cC[e];
        if (sup) sup[e] = s;
        if (live) {
            live[e] = s;
            rnd[e] = -1;
        }
        acc += s;
    }
    if (code)
        for (int64_t i = tid; i < E / 8 + 1; i += nth) code[i] = ~0u;
    acc = warp_sum(acc);
    if (lane_id() == 0) s_part[threadIdx.x / kWarp] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        long long b = 0;
        for (int i = 0; i < (int)(blockDim.x / kWarp); i++) b += s_part[i];
        atomicAdd((unsigned long long*)&ctl->triangles, (unsigned long long)b);
        if (!live) {
            __threadfence();
            if (atomicAdd(&ctl->done, 1u) == gridDim.x - 1) {
                for (int i = 0; i < TDT_STAT_COUNT; i++) stats[i] = 0;
                stats[TDT_STAT_STATUS] = *(volatile int*)&ctl->g.status;
                stats[TDT_STAT_TRIANGLES] = (long long)atomicAdd((unsigned long long*)&ctl->triangles, 0ull) / 3;
            }
        }
    }
}

// Truss numbers, and the digit totals of the sort by round.
__global__ void __launch_bounds__(256) truss_out_kernel(const int32_t* __restrict__ rnd,
                                                        const int32_t* __restrict__ round_level, int64_t E,
                                                        int32_t* __restrict__ truss, int passes, uint32_t* hist,
                                                        PeelCtl* ctl) {
    __shared__ uint32_t s_hist[kMaxPasses * kRadix];
    if (__syncthreads_or(*(volatile int*)&ctl->g.status != 0)) return;
    const int run = radix_passes_run(passes, ctl->rounds);
    DigitHist H{s_hist};
    H.init(run);
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < E;
         e += (int64_t)gridDim.x * blockDim.x) {
        const int32_t r = rnd[e];
        H.add((uint32_t)r, run);
        if (r < 0) {  // every edge is peeled when the run completes
            atomicMax((int*)&ctl->g.status, (int)TDT_ERR_CAPACITY);
            continue;
        }
        if (truss) truss[e] = __ldg(round_level + r) + 2;
    }
    H.flush(run, hist);
}

// Number of sorted positions whose round has level <= lv: the first round above
// it (levels do not fall from round to round), then its first position.
__device__ __forceinline__ int64_t count_level_le(const uint32_t* keys, int64_t E, const int32_t* round_level,
                                                  int64_t rounds, int32_t lv) {
    int64_t lo = 0, hi = rounds;
    while (lo < hi) {
        const int64_t mid = (lo + hi) >> 1;
        if (__ldg(round_level + mid) <= lv) lo = mid + 1; else hi = mid;
    }
    const int64_t r = lo;
    for (lo = 0, hi = E; lo < hi;) {
        const int64_t mid = (lo + hi) >> 1;
        if ((int64_t)__ldg(keys + mid) < r) lo = mid + 1; else hi = mid;
    }
    return lo;
}

// Stats words of a finished peel (how it found the triangles).
__device__ __forceinline__ void write_stats(const PeelCtl* ctl, int64_t* stats, int status) {
    for (int i = 0; i < TDT_STAT_COUNT; i++) stats[i] = 0;
    stats[TDT_STAT_STATUS] = status;
    stats[TDT_STAT_LISTED] = ctl->listed ? (ctl->compact_skip ? 1 : 2) : 0;
}

__global__ void ptr_etruss_kernel(const uint32_t* __restrict__ k0, const uint32_t* __restrict__ v0,
                                  const uint32_t* __restrict__ k1, const uint32_t* __restrict__ v1, int passes,
                                  int64_t E, const int32_t* __restrict__ round_level, int32_t* __restrict__ ptr_truss,
                                  int64_t ptr_cap, int32_t* __restrict__ e_truss, PeelCtl* ctl,
                                  int64_t* __restrict__ stats) {
    const int64_t tid = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int64_t nth = (int64_t)gridDim.x * blockDim.x;
    const int status = *(volatile int*)&ctl->g.status;
    if (status != 0) {  // of an earlier kernel, or thread 0's of this one
        if (tid == 0) write_stats(ctl, stats, status);
        return;
    }
    const long long rounds = ctl->rounds;
    const bool first = radix_passes_run(passes, rounds) & 1;
    const uint32_t* keys = first ? k0 : k1;
    const uint32_t* vals = first ? v0 : v1;
    const int32_t L = rounds > 0 ? round_level[rounds - 1] : 0;
    const int64_t n0 = rounds > 0 ? count_level_le(keys, E, round_level, rounds, 0) : E;
    if (ptr_truss) {
        if ((int64_t)L + 1 > ptr_cap) {
            if (tid == 0) atomicMax(&ctl->g.status, (int)TDT_ERR_CAPACITY);
        } else {
            for (int64_t i = tid; i <= L; i += nth)
                ptr_truss[i] = (int32_t)((i == 0 ? n0 : count_level_le(keys, E, round_level, rounds, (int32_t)i)) -
                                         n0);
        }
    }
    if (e_truss)
        for (int64_t p = n0 + tid; p < E; p += nth) e_truss[p - n0] = (int32_t)vals[p];
    if (tid == 0) {
        write_stats(ctl, stats, ptr_truss && (int64_t)L + 1 > ptr_cap ? TDT_ERR_CAPACITY : TDT_OK);
        stats[TDT_STAT_KMAX] = (long long)L + 2;
        stats[TDT_STAT_NPTR] = (long long)L + 1;
        stats[TDT_STAT_ROUNDS] = rounds;
        stats[TDT_STAT_TRIANGLES] = ctl->triangles / 3;
        stats[TDT_STAT_NETRUSS] = E - n0;
    }
}

// Membership; the last block writes the stats.
__global__ void ktruss_out_kernel(const int32_t* __restrict__ rnd, int64_t E, uint8_t* __restrict__ in_k,
                                  PeelCtl* ctl, int64_t* __restrict__ stats) {
    __shared__ unsigned long long s_part[32];
    unsigned long long acc = 0;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < E;
         e += (int64_t)gridDim.x * blockDim.x) {
        const uint8_t a = rnd[e] == -1;
        in_k[e] = a;
        acc += a;
    }
    acc = warp_sum(acc);
    if (lane_id() == 0) s_part[threadIdx.x / kWarp] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long b = 0;
        for (int i = 0; i < (int)(blockDim.x / kWarp); i++) b += s_part[i];
        atomicAdd(&ctl->alive, b);
        __threadfence();
        if (atomicAdd(&ctl->done, 1u) == gridDim.x - 1) {
            write_stats(ctl, stats, *(volatile int*)&ctl->g.status);
            stats[TDT_STAT_ALIVE] = (long long)atomicAdd(&ctl->alive, 0ull);
            stats[TDT_STAT_ROUNDS] = ctl->rounds;
            stats[TDT_STAT_TRIANGLES] = ctl->triangles / 3;
        }
    }
}

// ------------------------------------------------------------------ host side
constexpr int64_t kSearchNextEdges = 1 << 20;

void prof_mark(int phase, cudaStream_t st);

// Test hook: wall-clock budget of the next peel launches (<= 0: the default).
static long long g_peel_deadline_ns = 0;
void set_peel_deadline(long long ns) { g_peel_deadline_ns = ns; }

// Test hook: lower the k-truss collection batch limits (<= 0: the defaults).
static long long g_dyn_min_slots = 0;

// Block 0's clock of the last persistent peel run in this workspace (the
// control block sits at its start): processing, grid-barrier waits after
// processing, level changes, and the whole kernel, in ns.
int peel_clock(const void* ws, long long* ns, cudaStream_t st) {
    TDT_CHECK_ARG(ws != nullptr && ns != nullptr, "null pointer");
    const PeelCtl* ctl = reinterpret_cast<const PeelCtl*>(ws);
    unsigned long long t[4];
    TDT_CUDA(cudaMemcpyAsync(t, &ctl->t_proc, sizeof(t), cudaMemcpyDeviceToHost, st));
    TDT_CUDA(cudaStreamSynchronize(st));
    for (int i = 0; i < 4; i++) ns[i] = (long long)t[i];
    return TDT_OK;
}
void set_peel_dyn_min(long long slots) { g_dyn_min_slots = slots; }
// Peel grid in half-SM units (0: the size heuristic below); the autotuner's
// launch-shape dimension.
static int g_peel_half_sms = 0;
void set_peel_grid(int half_sms) { g_peel_half_sms = half_sms > 0 ? half_sms : 0; }
static long long g_fixed_item_cap = 0, g_fixed_cand_cap = 0;
void set_fixed_caps(long long items, long long cands) {
    g_fixed_item_cap = items;
    g_fixed_cand_cap = cands;
}

// The peel's barrier with one block that never reaches it: the others wait
// limit_ns, then leave with TDT_ERR_TIMEOUT in the status (the test of the
// bounded waits).
__global__ void barrier_probe_kernel(PeelCtl* ctl, unsigned long long limit_ns) {
    __shared__ RoundShared s_round;
    if (blockIdx.x == 0) return;
    if (threadIdx.x == 0) s_round.dmin = INT32_MAX;
    RoundBar RB{gridDim.x, 0ull, 0ull};
    round_barrier(ctl, RB, &s_round, 0, &ctl->dmin[0], limit_ns);
}

int test_barrier_timeout(void* ws, long long limit_ns, cudaStream_t st) {
    TDT_CHECK_ARG(ws != nullptr, "null workspace");
    TDT_CHECK_ARG(limit_ns >= 1000000ll && limit_ns <= 2000000000ll, "limit %lld ns outside [1 ms, 2 s]",
                  limit_ns);
    static_assert(sizeof(PeelCtl) <= 4096, "the probe's workspace");
    PeelCtl* ctl = reinterpret_cast<PeelCtl*>(ws);
    TDT_CUDA(cudaMemsetAsync(ctl, 0, sizeof(PeelCtl), st));
    barrier_probe_kernel<<<8, 32, 0, st>>>(ctl, (unsigned long long)limit_ns);
    TDT_LAUNCH_CHECK("barrier_probe");
    int status = 0;
    TDT_CUDA(cudaMemcpyAsync(&status, &ctl->g.status, sizeof(int), cudaMemcpyDeviceToHost, st));
    TDT_CUDA(cudaStreamSynchronize(st));
    return status;
}

int launch_walk_count(const int64_t* rp, const int32_t* cols, const int64_t* cp, const int32_t* in_src,
                      const int32_t* in_eid, int64_t nv, int64_t ne, int32_t* cA, int32_t* cB, int32_t* cC,
                      const int64_t* sbase, int2* stage_end, unsigned long long stage_slots, int* stage_skip,
                      int32_t* runA, void* units, void* longs, void* ctl, int* status, cudaStream_t st);
int launch_walk_list(const int64_t* rp, const int32_t* cols, const int64_t* cp, const int32_t* in_src,
                     const int32_t* in_eid, int64_t nv, int64_t ne, const int64_t* off, int32_t* cA, int2* lists,
                     int32_t* runA, void* units, void* longs, void* ctl, const int* gate, int* status, cudaStream_t st);
int launch_distribute(const int64_t* rp, const int32_t* cols, const int32_t* rows, const int64_t* cp,
                      const int32_t* in_eid, int64_t nv, int64_t ne, const int64_t* off, const int32_t* cA,
                      const int32_t* cB, const int64_t* sbase, const int2* stage_end, const int* stage_skip,
                      int2* lists, uint32_t* cnt, void* units, void* ctl, const int* gate, int* status,
                      cudaStream_t st);

namespace {
struct Carver {
    char* base;
    size_t off = 0;
    size_t cap;
    void* take(size_t bytes) {
        off = (off + 255) & ~(size_t)255;
        void* p = base ? base + off : nullptr;
        off += bytes;
        return p;
    }
};

struct Layout {
    PeelCtl* ctl;
    void* sup_ctl;
    int32_t* rows_d;
    int32_t* indeg;
    int64_t* cp;
    int32_t* in_src;
    int32_t* in_eid;
    int32_t* sup;
    int32_t* live;
    int32_t* rnd;
    int32_t* round_level;
    int4* qi[3];
    long long* qb[3];
    int64_t* off;
    int64_t* sbase;
    int32_t* sidx;
    int32_t* alive[2];
    unsigned* code;
    void* scan_cp;
    void* scan_sb;
    void* scan_off;
    void* sort_ws;
    size_t zero_count, zero_peel, zero_sort;
    size_t total;
};

Layout carve(void* ws, int64_t V, int64_t E) {
    Carver c{reinterpret_cast<char*>(ws)};
    Layout L;
    const size_t e = (size_t)(E > 0 ? E : 1), v = (size_t)(V > 0 ? V : 1);
    // zeroed at the start of a run, in one go: up to zero_count without a list tail
    // (three role counts an edge), to zero_peel with one (and the distribution's
    // counters), to zero_sort for a decomposition
    L.ctl = (PeelCtl*)c.take(4096);
    L.sup_ctl = c.take(256);
    L.scan_cp = c.take(scan_scratch_bytes((int64_t)v));
    L.scan_sb = c.take(scan_scratch_bytes((int64_t)v));
    L.scan_off = c.take(scan_scratch_bytes((int64_t)e));
    L.indeg = (int32_t*)c.take(4 * v);
    L.qi[0] = (int4*)c.take(16 * e);
    L.zero_count = c.off - 4 * e;
    L.zero_peel = c.off;
    L.sort_ws = c.take(radix_scratch(nullptr, (int64_t)e, 4).bytes);
    L.zero_sort = c.off;
    L.rows_d = (int32_t*)c.take(4 * e);
    L.cp = (int64_t*)c.take(8 * (v + 1));
    L.in_src = (int32_t*)c.take(4 * e);
    L.in_eid = (int32_t*)c.take(4 * e);
    L.sup = (int32_t*)c.take(4 * e);
    L.live = (int32_t*)c.take(4 * e);
    L.rnd = (int32_t*)c.take(4 * e);
    L.round_level = (int32_t*)c.take(4 * (e + 2));
    L.qb[0] = (long long*)c.take(8 * e);
    for (int b = 1; b < 3; b++) {
        L.qi[b] = (int4*)c.take(16 * e);
        L.qb[b] = (long long*)c.take(8 * e);
    }
    L.off = (int64_t*)c.take(8 * (e + 1));
    L.sbase = (int64_t*)c.take(8 * (v + 1));
    L.sidx = (int32_t*)c.take(8 * (size_t)kSlotIdx);
    L.alive[0] = (int32_t*)c.take(4 * e);
    L.alive[1] = (int32_t*)c.take(4 * e);
    L.code = (unsigned*)c.take(4 * (e / 8 + 1));
    L.total = c.off + 256;
    return L;
}
}  // namespace

size_t decompose_workspace_bytes(int64_t V, int64_t E) {
    // the e_truss sort reuses the queue buffers for its keys/values
    return carve(nullptr, V, E).total;
}

// mode 0: decomposition; 1: k-truss search at level fixed_level; 2: support / triangle count only.
int run_peel(int mode, const int32_t* rows, const int32_t* cols, const int64_t* rp, int64_t V, int64_t E,
             int32_t fixed_level, int32_t* truss, int32_t* e_truss, int32_t* ptr_truss, int64_t ptr_cap,
             uint8_t* in_k, int32_t* support_out, int64_t* stats, void* ws, size_t ws_bytes, cudaStream_t st) {
    TDT_CHECK_ARG(V >= 0 && E >= 0, "negative graph size");
    TDT_CHECK_ARG(E < (int64_t)INT32_MAX, "num_edges %lld exceeds int32 edge ids", (long long)E);
    TDT_CHECK_ARG(V < (int64_t)INT32_MAX, "num_vertices %lld exceeds int32 vertex ids", (long long)V);
    TDT_CHECK_ARG(stats != nullptr, "stats is required");
    TDT_CHECK_ARG(E == 0 || (cols && rp), "null graph pointer");
    const size_t need = decompose_workspace_bytes(V, E);
    if (ws_bytes < need || ws == nullptr) {
        set_error("workspace of %zu bytes < required %zu", ws_bytes, need);
        return TDT_ERR_WORKSPACE;
    }
    DeviceInfo di;
    int rc = device_info(&di);
    if (rc) return rc;
    Layout L = carve(ws, V, E);
    // The list tail: final lists grow from its start, the staging slots of the
    // one walk end at its end.
    const size_t list_base = (need + 255) & ~(size_t)255;
    const unsigned long long tail =
        mode != 2 && ws_bytes > list_base ? (unsigned long long)(ws_bytes - list_base) : 0ull;
    const size_t zero = mode == 0 ? L.zero_sort : tail > 0 ? L.zero_peel : L.zero_count;
    TDT_CUDA(cudaMemsetAsync(ws, 0, E == 0 ? 4096 : zero, st));
    if (E == 0) {
        TDT_CUDA(cudaMemsetAsync(stats, 0, sizeof(int64_t) * TDT_STAT_COUNT, st));
        if (mode == 0) {
            if (ptr_truss && ptr_cap >= 1) TDT_CUDA(cudaMemsetAsync(ptr_truss, 0, 4, st));
            int64_t h[TDT_STAT_COUNT] = {0, 2, 1, 0, 0, 0, 0, 0};
            if (ptr_truss && ptr_cap < 1) h[0] = TDT_ERR_CAPACITY;
            TDT_CUDA(cudaMemcpyAsync(stats, h, sizeof(h), cudaMemcpyHostToDevice, st));
            TDT_CUDA(cudaStreamSynchronize(st));
        }
        return TDT_OK;
    }
    const int tb = 256;
    const unsigned g_e = grid_for(E, tb, di.sms, 8);
    const int32_t* rows_use = rows ? rows : L.rows_d;
    if (rows)
        validate_kernel<<<g_e, tb, 0, st>>>(rp, rows, cols, E, V, L.ctl);
    else
        validate_rows_kernel<<<grid_for(V * 32, kValBlock, di.sms, 8), kValBlock, 0, st>>>(rp, L.rows_d, cols, E, V, L.ctl);
    TDT_LAUNCH_CHECK("validate");
    // cA, cB, cC (role counts) live in the first queue buffer until the peel starts
    int32_t* cA = reinterpret_cast<int32_t*>(L.qi[0]);
    int32_t* cB = cA + E;
    int32_t* cC = cB + E;
    int2* lists = reinterpret_cast<int2*>(reinterpret_cast<char*>(ws) + list_base);
    int2* stage_end = lists + tail / 8;
    prof_mark(0, st);
    // in-adjacency (CSC) of the oriented graph: the walk's middle vertices, and
    // the peel without lists
    // tiles of the in-adjacency build: at least one per resident block
    const int64_t csc_blocks = (int64_t)di.sms * 4;
    int64_t csc_tile = kCscTile;
    while (csc_tile > 1024 && E < csc_tile * csc_blocks) csc_tile /= 2;
    const int64_t csc_tiles = (E + csc_tile - 1) / csc_tile;
    const unsigned g_csc = (unsigned)(csc_tiles < csc_blocks ? csc_tiles : csc_blocks);
    indeg_kernel<<<g_csc, kCscBlock, 0, st>>>(cols, E, V, L.indeg, L.ctl);
    TDT_LAUNCH_CHECK("indeg");
    rc = tail > 0 ? scan_rows(L.indeg, L.cp, L.scan_cp, rp, L.sbase, L.scan_sb, V, &L.ctl->g.status, st)
                  : exclusive_scan(L.indeg, L.cp, V, L.cp + V, L.scan_cp, &L.ctl->g.status, st);
    if (rc) return rc;
    csc_fill_kernel<<<g_csc, kCscBlock, 0, st>>>(rows_use, cols, E, V, csc_tile, L.cp, L.indeg, L.in_src, L.in_eid, L.ctl);
    TDT_LAUNCH_CHECK("csc_fill");
    // the walk: counts, and the role-A entries when they can be staged (skipped
    // on the device when validation failed); the plan of its units stays for
    // the list walk
    rc = launch_walk_count(rp, cols, L.cp, L.in_src, L.in_eid, V, E, cA, cB, cC, tail > 0 ? L.sbase : nullptr,
                           stage_end, tail / 8, &L.ctl->stage_skip, L.alive[0], L.qi[2], L.qi[1], L.sup_ctl,
                           &L.ctl->g.status, st);
    if (rc) return rc;
    const bool peel = mode != 2;
    init_state_kernel<<<g_e, tb, 0, st>>>(cA, cB, cC, peel ? L.sup : support_out, peel ? L.live : nullptr, L.rnd,
                                          peel ? L.code : nullptr, E, L.ctl, stats);
    TDT_LAUNCH_CHECK("init_state");
    prof_mark(1, st);
    if (mode == 2) {
        for (int ph = 2; ph <= 4; ph++) prof_mark(ph, st);
        return TDT_OK;
    }
    // per-edge triangle lists in the workspace tail when 24 T bytes fit
    if (tail > 0) {
        const ListDecision D{L.sbase + V, tail, &L.ctl->stage_skip, &L.ctl->listed, &L.ctl->list_skip,
                             &L.ctl->compact_skip, &L.ctl->rewalk_skip};
        rc = scan_lists(L.sup, L.off, E, L.scan_off, D, &L.ctl->g.status, st);
        if (rc) return rc;
        // second walk, when the lists fit but not beside the staging slots
        rc = launch_walk_list(rp, cols, L.cp, L.in_src, L.in_eid, V, E, L.off, cA, lists, L.alive[0], L.qi[2],
                              L.qi[1], L.sup_ctl, &L.ctl->rewalk_skip, &L.ctl->g.status, st);
        if (rc) return rc;
        rc = launch_distribute(rp, cols, rows_use, L.cp, L.in_eid, V, E, L.off, cA, cB, L.sbase, stage_end,
                               &L.ctl->compact_skip, lists, reinterpret_cast<uint32_t*>(cC + E), L.qi[2], L.sup_ctl, &L.ctl->list_skip, &L.ctl->g.status, st);
        if (rc) return rc;
    }
    prof_mark(2, st);

    // persistent peel
    PeelArgs A;
    A.rp = rp; A.cols = cols; A.rows = rows_use; A.cp = L.cp; A.in_src = L.in_src; A.in_eid = L.in_eid;
    A.live = L.live; A.rnd = L.rnd; A.round_level = L.round_level;
    for (int b = 0; b < 3; b++) {
        A.qi[b] = L.qi[b];
        A.qb[b] = L.qb[b];
    }
    A.code = L.code;
    A.off = L.off; A.lists = lists;
    // the search peel's copy of the out-edges and the row lengths, in arrays
    // that only the listing uses
    A.out_col = reinterpret_cast<int32_t*>(L.off);
    A.out_eid = A.out_col + E;
    A.out_len = reinterpret_cast<int32_t*>(L.sbase);
    A.in_len = L.indeg;
    A.alive[0] = L.alive[0]; A.alive[1] = L.alive[1];
    A.sidx[0] = L.sidx; A.sidx[1] = L.sidx + kSlotIdx;
    A.V = V; A.E = E; A.round_cap = E + 2;
    A.mode = mode == 0 ? 0 : 1;
    A.fixed_level = fixed_level;
    A.deadline_ns = g_peel_deadline_ns > 0 ? (unsigned long long)g_peel_deadline_ns : kPeelDeadlineNs;
    A.dyn_min_slots = g_dyn_min_slots > 0 ? g_dyn_min_slots : (1ll << kDynMinLog2);
    A.fixed_item_cap = g_fixed_item_cap > 0 && (unsigned long long)g_fixed_item_cap < kFixedItemCap
                           ? (unsigned long long)g_fixed_item_cap : kFixedItemCap;
    A.fixed_cand_cap = g_fixed_cand_cap > 0 && (unsigned long long)g_fixed_cand_cap < kFixedCandCap
                           ? (unsigned long long)g_fixed_cand_cap : kFixedCandCap;
    A.ctl = L.ctl;
    // Small graphs peel their lists on one block per SM: their sub-rounds fit
    // one window a warp there, and a grid barrier of fewer blocks is shorter.
    // 76 / 152 / 304 blocks: R-MAT scale 12 1.77 / 1.80 / 1.92 ms, scale 14
    // 4.42 / 4.36 / 4.64, scale 16 (0.9 M edges) 8.43 / 7.53 / 7.52, scale 18
    // 18.2 / 14.0 / 13.3, scale 20 61.4 / 40.2 / 34.1; Chung-Lu (1.5 M edges)
    // 10.6 / 9.6 / 9.8.  The search peel keeps every block: its slots are
    // binary searches.
    // With a list tail the device decides whether the peel is listed.  A large
    // graph whose lists do not fit then goes to the compacting search kernel,
    // which follows (a launch that returns at once costs 4 us); a small one is
    // searched in place.
    A.search_next = mode == 0 && tail > 0 && E >= kSearchNextEdges;
    auto launch_peel = [&](void* kern, bool lists_k) -> int {
        int occ = 0;
        TDT_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, kPeelBlock, 0));
        if (occ < 1) {
            set_error("peel kernel cannot be resident");
            return TDT_ERR_UNSUPPORTED;
        }
        if (di.sms * occ > 4096) occ = 4096 / di.sms;
        int nblk = di.sms * occ;
        if (lists_k && E < (1ll << 20)) nblk = di.sms;
        if (g_peel_half_sms > 0) nblk = (g_peel_half_sms * di.sms + 1) / 2;
        if (nblk > di.sms * occ) nblk = di.sms * occ;
        void* args[] = {&A};
        TDT_CUDA(cudaLaunchCooperativeKernel(kern, dim3(nblk), dim3(kPeelBlock), args, 0, st));
        note_launch();
        return TDT_OK;
    };
    if (tail > 0) rc = launch_peel((void*)peel_kernel<kListed>, true);
    if (rc == TDT_OK && (tail == 0 || A.search_next))
        rc = launch_peel(mode == 0 ? (void*)peel_kernel<kCompact> : (void*)peel_kernel<kSearch>, false);
    if (rc) return rc;
    prof_mark(3, st);

    if (mode == 0) {
        // outputs: truss numbers, then e_truss / ptr_truss from a stable sort of
        // the edges by round (as many passes as the rounds have digits)
        uint32_t* k0 = reinterpret_cast<uint32_t*>(L.qi[0]);
        uint32_t* v0 = k0 + E;
        uint32_t* k1 = reinterpret_cast<uint32_t*>(L.qi[1]);
        uint32_t* v1 = k1 + E;
        int passes = 1;
        while (passes < 4 && ((int64_t)1 << (8 * passes)) < E + 2) passes++;
        const RadixScratch R = radix_scratch(L.sort_ws, E, passes);
        truss_out_kernel<<<g_e, tb, 0, st>>>(L.rnd, L.round_level, E, truss, passes, R.hist, L.ctl);
        TDT_LAUNCH_CHECK("truss_out");
        rc = radix_sort<uint32_t, true>(reinterpret_cast<const uint32_t*>(L.rnd), k0, k1, v0, v1, E, passes, R, nullptr,
                                        &L.ctl->rounds, &L.ctl->g.status, st);
        if (rc) return rc;
        ptr_etruss_kernel<<<g_e, tb, 0, st>>>(k0, v0, k1, v1, passes, E, L.round_level, ptr_truss, ptr_cap, e_truss,
                                              L.ctl, stats);
        TDT_LAUNCH_CHECK("ptr_etruss");
    } else {
        ktruss_out_kernel<<<g_e, tb, 0, st>>>(L.rnd, E, in_k, L.ctl, stats);
        TDT_LAUNCH_CHECK("ktruss_out");
    }
    prof_mark(4, st);
    return TDT_OK;
}

}  // namespace tdt
