// The drop-in support operator: per-edge support over a CSR of any acyclic
// orientation, without scratch memory.
//
// Replaces checkElementsTwoPtr / checkElementsTwoPtrTile (kernel.cu:28-141),
// which give every edge (u,v) one thread that merges N+(u) and N+(v) and adds
// +1 to (u,w), +1 to (v,w) and +count to (u,v) for every common w.
//
// Here the unit of work is the source vertex u of the triangle (u, v, w)
// (u -> v, u -> w, v -> w):
//   * N+(u) is staged once in shared memory (one warp for d+(u) <= warp_cap,
//     a whole block for larger rows; rows beyond the block buffer are searched
//     in place), with a bitmap of its hashed vertex ids;
//   * the wedges (v, w), v in N+(u), w in N+(v), form one flat index space
//     (the out-lists of a group of v's back to back: 32 v's for a warp, 512 for
//     a block).  A warp walks it 32 consecutive wedges per step (coalesced
//     loads of N+(v)); the owner v of each lane's wedge comes from one
//     OR-reduction of the group boundaries inside the step, not a search;
//   * w is tested against the bitmap; most wedges close no triangle and stop
//     there.  Candidates go to a per-warp queue in shared memory and are
//     resolved 32 at a time by binary search in N+(u) (full warps instead of a
//     few active lanes);
//   * hits on (u,v) and (u,w) go to shared-memory counters flushed once per
//     row; only the (v,w) hit is a global atomic.
// Each triangle is found exactly once, from its (source, middle) edge, so the
// counts are the reference's for any n_cut.  The whole-path calls, which keep
// an in-adjacency, walk from the middle vertex instead (walk.cu).
#include "common.cuh"

namespace tdt {

constexpr int kSupBlock = 512;                 // 16 warps
constexpr int kSupWarps = kSupBlock / kWarp;
#ifndef TDT_SUP_MINB
#define TDT_SUP_MINB 3
#endif
constexpr int kSupMinBlocks = TDT_SUP_MINB;    // resident blocks per SM (3: registers <= 42)
constexpr int kSupSmemBytes = 64 * 1024;       // dynamic shared memory per block
constexpr int kVertexBatch = 2;                // light vertices per turn below the top quarter of ids
constexpr int kQueue = 64;                     // candidate queue entries per warp

// Light rows: one warp, a 4 KB slice of the block buffer:
//   su[256] | cnt[256] | group S[32] VI[32] BV[32] | bitmap 8192 bits | queue
constexpr int kWarpCap = 256;
constexpr int kSliceBytes = kSupSmemBytes / kSupWarps;
constexpr int kLightBmLog2 = 13;
constexpr int kSlSu = 0;
constexpr int kSlCnt = kSlSu + 4 * kWarpCap;
constexpr int kSlS = kSlCnt + 4 * kWarpCap;
constexpr int kSlVI = kSlS + 4 * kWarp;
constexpr int kSlBV = kSlVI + 4 * kWarp;
constexpr int kSlBm = kSlBV + 8 * kWarp;
constexpr int kSlQ = kSlBm + (1 << kLightBmLog2) / 8;
static_assert(kSlQ + 8 * kQueue <= kSliceBytes, "light slice");
// a push adds up to 32 candidates to a queue holding up to 31 (it is drained
// to below 32 after every push)
static_assert(kQueue >= 2 * kWarp, "candidate queue");
// the vectorised walk keeps a group as int4 {SC, BV, HI, VI} over S|VI|BV|HI
static_assert(kSlS % 16 == 0 && kSlVI == kSlS + 4 * kWarp && kSlBV == kSlVI + 4 * kWarp && kSlBm >= kSlS + 16 * kWarp,
              "light group layout");

// Heavy rows: one block, the whole buffer:
//   su[H] | cnt[H] | group S[512] VI[512] BV[512] | bitmap 2^16 bits | queues
// Rows longer than H are searched in place (su and counters in global memory)
// with a 2^18-bit bitmap over the su/cnt area.
constexpr int kSeg = kSupBlock;                // v's per heavy group (one per thread)
constexpr int kHeavyBmLog2 = 16;
constexpr int kHugeBmLog2 = 18;
constexpr int kHvQueues = kSupSmemBytes - kSupWarps * 8 * kQueue;
constexpr int kHvBm = kHvQueues - (1 << kHeavyBmLog2) / 8;
constexpr int kHvBV = kHvBm - 8 * kSeg;
constexpr int kHvVI = kHvBV - 4 * kSeg;
constexpr int kHvS = kHvVI - 4 * kSeg;
constexpr int kHeavyCap = kHvS / 8;            // su + cnt, 8 bytes per entry
static_assert(kHeavyCap >= 4096, "heavy cap");
static_assert(kHvS % 16 == 0 && kHvVI == kHvS + 4 * kSeg && kHvBV == kHvVI + 4 * kSeg && kHvBm >= kHvS + 16 * kSeg,
              "heavy group layout");
static_assert((1 << kHugeBmLog2) / 8 <= kHvS, "in-place bitmap");

// Row ranges are clamped to [0, ne] so a malformed row_ptr cannot move an
// access outside cols/out.
struct OutRows {
    const int32_t* rp;
    int32_t stride;  // row_ptr entries per vertex (n_cut)
    const int32_t* cols;
    int64_t nv;      // vertices
    int64_t ne;      // edges
    __device__ __forceinline__ int32_t clamp(int32_t x) const { return x < 0 ? 0 : (x > ne ? (int32_t)ne : x); }
    __device__ __forceinline__ int32_t begin(int64_t v) const { return clamp(__ldg(rp + v * stride)); }
    __device__ __forceinline__ int32_t end(int64_t v) const {
        const int32_t b = begin(v), e = clamp(__ldg(rp + v * stride + stride));
        return e < b ? b : e;
    }
};

struct SupArgs {
    int32_t* out;
    int warp_cap;                   // rows with d+ <= warp_cap go to one warp (<= kWarpCap)
    int heavy_cap;                  // heavier rows staged in smem up to this size (<= kHeavyCap)
};

// Test hook: lower the light/heavy thresholds so small graphs drive every path
// (0 restores the defaults).
static int g_warp_cap = 0, g_heavy_cap = 0;
// Test hook: 0 forces the scalar wedge walk (the vectorised one is the default).
static int g_vec_walk = 1;
void set_vector_walk(int on) { g_vec_walk = on != 0; }
void set_support_caps(int warp_cap, int heavy_cap) {
    g_warp_cap = warp_cap;
    g_heavy_cap = heavy_cap;
}

void support_caps(int* warp_cap, int* heavy_cap) {
    *warp_cap = g_warp_cap;
    *heavy_cap = g_heavy_cap;
}

#ifndef TDT_BM_LOWBITS
#define TDT_BM_LOWBITS 1
#endif
// Bitmap index of vertex id w: its low bits (ids are degree ranks, and a
// row's out-neighbours cluster among the high ranks, so consecutive ids land
// on distinct bits), or a multiplicative hash.
__device__ __forceinline__ uint32_t bm_hash(int32_t w, int log2bits) {
    if (TDT_BM_LOWBITS) return (uint32_t)w & ((1u << log2bits) - 1u);
    return ((uint32_t)w * 0x9E3779B1u) >> (32 - log2bits);
}

// Binary search of key in s[lo, hi) (shared or global, generic address).
__device__ __forceinline__ int bsearch_i32(const int32_t* s, int lo, int hi, int32_t key) {
    int end = hi;
    while (lo < hi) {
        int mid = (lo + hi) >> 1;
        if (s[mid] < key) lo = mid + 1; else hi = mid;
    }
    return (lo < end && s[lo] == key) ? lo : -1;
}

// One staged row.  packed: counts in shared memory; otherwise added to the
// output directly.
struct RowState {
    const int32_t* su;            // N+(u)
    uint32_t* cnt;
    const uint32_t* bm;           // bitmap of hashed N+(u)
    int bm_log2;
    int d;
    int32_t umax;                 // largest id in N+(u)
    bool packed;
    int32_t bu;                   // position of the row's first edge
};

// One triangle (u, v = su[i], w = su[p]) with (v,w) at position pos.
__device__ __forceinline__ void on_triangle(const RowState& R, const SupArgs& A, int i, int p, int32_t pos) {
    if (R.packed) {
        atomicAdd(R.cnt + i, 1u);
        atomicAdd(R.cnt + p, 1u);
    } else {
        atomicAdd(A.out + R.bu + i, 1);
        atomicAdd(A.out + R.bu + p, 1);
    }
    atomicAdd(A.out + pos, 1);
}

// Per-warp candidate queue: wedge position (the (v,w) edge) and v's index i.
struct WarpQueue {
    int32_t* pos;
    int32_t* vi;
    int n;                        // warp-uniform fill
};

// Resolve queue entries [0, cnt) (cnt <= 32), one per lane.
__device__ __forceinline__ void resolve(const OutRows& G, const SupArgs& A, const RowState& R,
                                        const WarpQueue& Q, int cnt) {
    const unsigned lane = lane_id();
    if ((int)lane < cnt) {
        const int32_t pos = Q.pos[lane];
        const int i = Q.vi[lane];
        const int32_t w = __ldg(G.cols + pos);
        const int p = bsearch_i32(R.su, 0, R.d, w);
        if (p >= 0) on_triangle(R, A, i, p, pos);
    }
}

// Positions in cols are int32, as the operator's row_ptr.
//
// Walk wedges [w0, w1) of a group: S[0..n) are the strictly increasing starts
// of the group's non-empty out-lists in the flat wedge space, BV their
// positions in cols, VI the index of their v in N+(u).  w0 is a multiple of
// 32 and o0 the group entry that holds wedge w0.
__device__ __forceinline__ void walk_group(const OutRows& G, const SupArgs& A, const RowState& R,
                                           const int32_t* S, const int32_t* VI, const int32_t* BV, int n, int w0, int w1,
                                           int o0, WarpQueue& Q) {
    const unsigned lane = lane_id();
    const unsigned lt = lanemask_lt();
    int ob = o0;
    for (int base = w0; base < w1; base += kWarp) {
        // group starts inside (base, base + 32): each is > base, and at most 31 fit
        const int k = ob + 1 + (int)lane;
        const int32_t B = k < n ? S[k] : INT32_MAX;
        const unsigned bit = ((unsigned)(B - base) < (unsigned)kWarp) ? (1u << (B - base)) : 0u;
        const unsigned mk = __reduce_or_sync(kFull, bit);
        const int nb = __popc(mk);
        const int32_t Bn = __shfl_sync(kFull, B, nb);
        const int t = base + (int)lane;
        bool cand = false;
        int32_t pos32 = 0;
        int vi = 0;
        if (t < w1) {
            const int o = ob + __popc(mk & (lt | (1u << lane)));
            const int32_t pos = BV[o] + (t - S[o]);
            const int32_t w = __ldg(G.cols + pos);
            if (w <= R.umax) {
                const uint32_t h = bm_hash(w, R.bm_log2);
                cand = (R.bm[h >> 5] >> (h & 31)) & 1u;
            }
            pos32 = (int32_t)pos;
            vi = VI[o];
        }
        ob += nb + (Bn == base + kWarp ? 1 : 0);
        const unsigned cm = __ballot_sync(kFull, cand);
        if (cm) {
            if (cand) {
                const int at = Q.n + __popc(cm & lt);
                Q.pos[at] = pos32;
                Q.vi[at] = vi;
            }
            Q.n += __popc(cm);
            if (Q.n >= kWarp) {
                __syncwarp();
                resolve(G, A, R, Q, kWarp);
                __syncwarp();
                const int rest = Q.n - kWarp;
                int32_t p2 = 0, v2 = 0;
                if ((int)lane < rest) {
                    p2 = Q.pos[kWarp + lane];
                    v2 = Q.vi[kWarp + lane];
                }
                __syncwarp();
                if ((int)lane < rest) {
                    Q.pos[lane] = p2;
                    Q.vi[lane] = v2;
                }
                __syncwarp();
                Q.n = rest;
            }
        }
    }
}

// The same walk over 16-byte chunks of cols, four wedges per lane and step:
// each out-list N+(v) = cols[BV[k], HI[k]) is widened to the aligned chunks
// that hold it, so a chunk belongs to one v and comes with one int4 load; the
// widened ends are masked by [BV[k], HI[k]).  SC[0..n) are the strictly
// increasing chunk starts of the group's lists in the flat chunk space, c0 a
// multiple of 32 and o0 the group entry that holds chunk c0.  The group is
// one int4 per list, GE[k] = {SC[k], BV[k], HI[k], VI[k]}: a lane reads its
// list's entry with one shared-memory load.  One owner
// reduction serves 128 wedges instead of 32.  cols must be 16-byte aligned
// (a 16-byte chunk never crosses a page, so the widened reads stay mapped).
__device__ __forceinline__ void walk_group_vec(const OutRows& G, const SupArgs& A, const RowState& R,
                                               const int4* GE, int n, int c0, int c1, int o0, WarpQueue& Q) {
    const unsigned lane = lane_id();
    const unsigned lt = lanemask_lt();
    const int4* __restrict__ cols4 = reinterpret_cast<const int4*>(G.cols);
    int ob = o0;
    for (int base = c0; base < c1; base += kWarp) {
        const int k = ob + 1 + (int)lane;
        const int32_t B = k < n ? GE[k].x : INT32_MAX;
        const unsigned bit = ((unsigned)(B - base) < (unsigned)kWarp) ? (1u << (B - base)) : 0u;
        const unsigned mk = __reduce_or_sync(kFull, bit);
        const int nb = __popc(mk);
        const int32_t Bn = __shfl_sync(kFull, B, nb);
        const int c = base + (int)lane;
        unsigned cm = 0;
        int32_t p0 = 0;
        int vi = 0;
        if (c < c1) {
            const int o = ob + __popc(mk & (lt | (1u << lane)));
            const int4 ge = GE[o];
            const int32_t lo = ge.y, hi = ge.z;
            p0 = ((lo >> 2) + (c - ge.x)) << 2;
            const int4 w4 = __ldg(cols4 + (p0 >> 2));
            const int32_t wq[4] = {w4.x, w4.y, w4.z, w4.w};
            // the chunk's entries inside [lo, hi): a mask, once per chunk
            unsigned vm = 0xFu;
            if (p0 < lo) vm &= 0xFu << (lo - p0);
            if (p0 + 4 > hi) vm &= 0xFu >> (p0 + 4 - hi);
            // every entry is tested (a hashed index stays inside the bitmap)
            // and the mask applied after
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int32_t w = wq[q];
                const uint32_t h = bm_hash(w, R.bm_log2);
                const unsigned hit = (R.bm[h >> 5] >> (h & 31)) & (w <= R.umax ? 1u : 0u);
                cm |= hit << q;
            }
            cm &= vm;
            vi = ge.w;
        }
        ob += nb + (Bn == base + kWarp ? 1 : 0);
        if (__any_sync(kFull, cm != 0)) {
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const bool cand = (cm >> q) & 1u;
                const unsigned m = __ballot_sync(kFull, cand);
                if (m == 0) continue;
                if (cand) {
                    const int at = Q.n + __popc(m & lt);
                    Q.pos[at] = p0 + q;
                    Q.vi[at] = vi;
                }
                Q.n += __popc(m);
                if (Q.n >= kWarp) {
                    __syncwarp();
                    resolve(G, A, R, Q, kWarp);
                    __syncwarp();
                    const int rest = Q.n - kWarp;
                    int32_t p2 = 0, v2 = 0;
                    if ((int)lane < rest) {
                        p2 = Q.pos[kWarp + lane];
                        v2 = Q.vi[kWarp + lane];
                    }
                    __syncwarp();
                    if ((int)lane < rest) {
                        Q.pos[lane] = p2;
                        Q.vi[lane] = v2;
                    }
                    __syncwarp();
                    Q.n = rest;
                }
            }
        }
    }
}

__device__ __forceinline__ void drain(const OutRows& G, const SupArgs& A, const RowState& R, WarpQueue& Q) {
    __syncwarp();
    if (Q.n > 0) resolve(G, A, R, Q, Q.n);
    __syncwarp();
    Q.n = 0;
}

// Stage row u (d entries at bu).  in_smem: su and packed counters in the
// given buffers; otherwise the global arrays.  The bitmap (2^bm_log2 bits) is
// cleared and filled; block_sync selects block- or warp-wide synchronisation.
__device__ __forceinline__ RowState stage_row(const OutRows& G, const SupArgs& A, int32_t* su_buf,
                                              uint32_t* cnt_buf, uint32_t* bm, int bm_log2, bool in_smem, int32_t bu,
                                              int d, int tid, int nthr, bool block_sync) {
    RowState R;
    R.bu = bu;
    R.d = d;
    R.bm = bm;
    R.bm_log2 = bm_log2;
    R.packed = in_smem;
    for (int i = tid; i < (1 << bm_log2) / 32; i += nthr) bm[i] = 0u;
    if (block_sync) __syncthreads(); else __syncwarp();
    if (in_smem) {
        R.su = su_buf;
        R.cnt = cnt_buf;
        for (int i = tid; i < d; i += nthr) {
            const int32_t w = __ldg(G.cols + bu + i);
            su_buf[i] = w;
            cnt_buf[i] = 0u;
            const uint32_t h = bm_hash(w, bm_log2);
            atomicOr(bm + (h >> 5), 1u << (h & 31));
        }
    } else {
        R.su = G.cols + bu;
        R.cnt = nullptr;
        for (int i = tid; i < d; i += nthr) {
            const uint32_t h = bm_hash(__ldg(G.cols + bu + i), bm_log2);
            atomicOr(bm + (h >> 5), 1u << (h & 31));
        }
    }
    R.umax = d > 0 ? __ldg(G.cols + bu + d - 1) : INT32_MIN;
    return R;
}

__device__ __forceinline__ void flush_row(const RowState& R, const SupArgs& A, int tid, int nthr) {
    if (!R.packed) return;
    for (int i = tid; i < R.d; i += nthr)
        if (R.cnt[i]) atomicAdd(A.out + R.bu + i, (int32_t)R.cnt[i]);
}

// Schedule, without scratch memory: the rows are dealt out to the blocks, row
// after row, because rows next to each other cost alike (ids are degree ranks);
// the warps of a block take its light rows from a counter in shared memory.
// Against chunks of 16 rows next to each other (SMs active 55 % of the time):
// R-MAT scale 18 (3.8 M edges) 2.68 -> 1.34 ms, 20 (15.7 M) 9.9 -> 8.1, 300 K
// Chung-Lu vertices 1.23 -> 1.07.  Rows shared by the blocks of a cluster,
// from a counter in its first block: clusters of 2 / 4 / 8 1.33 / 1.36 / 1.47 ms
// at scale 18.  The rest is the walk: its bitmap tests and the wedge loads.
//
// kVec: the wedge walk loads 16-byte chunks of cols (walk_group_vec).
template <bool kVec>
__global__ void __launch_bounds__(kSupBlock, kSupMinBlocks) support_kernel(OutRows G, SupArgs A) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int32_t s_list[kSupBlock];
    __shared__ int32_t s_wsum[2][kSupWarps + 1];
    __shared__ int s_n;
    __shared__ unsigned s_light;
    const int wib = threadIdx.x / kWarp;
    const unsigned lane = lane_id();
    const int64_t nv = G.nv;
    const int64_t step = gridDim.x, first = blockIdx.x;
    const int64_t mine = first < nv ? (nv - first + step - 1) / step : 0;  // rows first, first + step, ..
    if (threadIdx.x == 0) s_light = 0;
    const int warp_cap = A.warp_cap;
    const int heavy_cap = A.heavy_cap;

    // ---- phase 1: rows with d+(u) > warp_cap, one block per row
    {
        int32_t* h_su = reinterpret_cast<int32_t*>(smem);
        uint32_t* h_cnt = reinterpret_cast<uint32_t*>(smem + 4 * kHeavyCap);
        int32_t* g_S = reinterpret_cast<int32_t*>(smem + kHvS);
        int32_t* g_VI = reinterpret_cast<int32_t*>(smem + kHvVI);
        int32_t* g_BV = reinterpret_cast<int32_t*>(smem + kHvBV);
        int32_t* g_HI = g_BV + kSeg;  // list ends (the vectorised walk)
        int4* g_GE = reinterpret_cast<int4*>(smem + kHvS);  // the vectorised walk's layout of the same area
        WarpQueue Q;
        Q.pos = reinterpret_cast<int32_t*>(smem + kHvQueues + wib * 8 * kQueue);
        Q.vi = Q.pos + kQueue;
        Q.n = 0;
        for (int64_t k0 = 0; k0 < mine; k0 += kSupBlock) {
            if (threadIdx.x == 0) s_n = 0;
            __syncthreads();
            const int64_t k = k0 + threadIdx.x;
            if (k < mine) {
                const int64_t u = first + k * step;
                if (G.end(u) - G.begin(u) > warp_cap) s_list[atomicAdd(&s_n, 1)] = (int32_t)u;
            }
            __syncthreads();
            const int nh = s_n;
            __syncthreads();  // every thread has read s_n before thread 0 resets it
            for (int h = 0; h < nh; h++) {
                const long long u = s_list[h];
                const int32_t bu = G.begin(u);
                const int d = (int)(G.end(u) - bu);
                const bool in_smem = d <= heavy_cap;
                uint32_t* bm = in_smem ? reinterpret_cast<uint32_t*>(smem + kHvBm) : reinterpret_cast<uint32_t*>(smem);
                RowState R = stage_row(G, A, h_su, h_cnt, bm, in_smem ? kHeavyBmLog2 : kHugeBmLog2, in_smem, bu, d,
                                       threadIdx.x, kSupBlock, true);
                __syncthreads();
                const int vend = d;
                for (int g0 = 0; g0 < vend; g0 += kSeg) {
                    // group: v's g0 .. g0+511, one per thread
                    const int i = g0 + threadIdx.x;
                    int32_t len = 0;
                    int32_t bv = 0;
                    if (i < vend) {
                        const int32_t v = R.su[i];
                        if (v >= 0 && v < nv) {
                            bv = (int32_t)G.begin(v);
                            len = (int32_t)(G.end(v) - bv);
                        }
                    }
                    // work units of the walk: wedges, or 16-byte chunks of cols
                    const int32_t units = kVec ? (len > 0 ? ((bv + len + 3) >> 2) - (bv >> 2) : 0) : len;
                    const unsigned nem = __ballot_sync(kFull, len > 0);
                    const int32_t incl = warp_incl_scan(units);
                    if (lane == 31) {
                        s_wsum[0][wib] = incl;
                        s_wsum[1][wib] = __popc(nem);
                    }
                    __syncthreads();
                    if (wib == 0) {
                        const int32_t x = (int)lane < kSupWarps ? s_wsum[0][lane] : 0;
                        const int32_t y = (int)lane < kSupWarps ? s_wsum[1][lane] : 0;
                        const int32_t xi = warp_incl_scan(x), yi = warp_incl_scan(y);
                        if ((int)lane < kSupWarps) {
                            s_wsum[0][lane] = xi - x;
                            s_wsum[1][lane] = yi - y;
                        }
                        if ((int)lane == kSupWarps - 1) {
                            s_wsum[0][kSupWarps] = xi;
                            s_wsum[1][kSupWarps] = yi;
                        }
                    }
                    __syncthreads();
                    if (len > 0) {
                        const int ci = s_wsum[1][wib] + __popc(nem & lanemask_lt());
                        if (kVec) {
                            g_GE[ci] = make_int4(s_wsum[0][wib] + incl - units, bv, bv + len, i);
                        } else {
                            g_S[ci] = s_wsum[0][wib] + incl - units;
                            g_VI[ci] = i;
                            g_BV[ci] = bv;
                            g_HI[ci] = bv + len;
                        }
                    }
                    const int total = s_wsum[0][kSupWarps];
                    const int n = s_wsum[1][kSupWarps];
                    __syncthreads();
                    // equal shares of the group's wedges, in whole steps of 32
                    const int share = ((total + kSupBlock - 1) / kSupBlock) * kWarp;
                    const int w0 = wib * share;
                    const int w1 = w0 + share < total ? w0 + share : total;
                    if (w0 < w1) {
                        int o0 = 0;
                        if (lane == 0) {
                            int lo = 0, hi = n - 1;  // last entry with S <= w0
                            while (lo < hi) {
                                const int mid = (lo + hi + 1) >> 1;
                                if ((kVec ? g_GE[mid].x : g_S[mid]) <= w0) lo = mid; else hi = mid - 1;
                            }
                            o0 = lo;
                        }
                        o0 = __shfl_sync(kFull, o0, 0);
                        if (kVec) walk_group_vec(G, A, R, g_GE, n, w0, w1, o0, Q);
                        else walk_group(G, A, R, g_S, g_VI, g_BV, n, w0, w1, o0, Q);
                    }
                    __syncthreads();  // the group arrays are rewritten next
                }
                drain(G, A, R, Q);
                __syncthreads();
                flush_row(R, A, threadIdx.x, kSupBlock);
                __syncthreads();
            }
        }
    }

    // ---- phase 2: rows with 2 <= d+(u) <= warp_cap, one warp per row
    __syncthreads();
    unsigned char* sl = smem + wib * kSliceBytes;
    int32_t* l_su = reinterpret_cast<int32_t*>(sl + kSlSu);
    uint32_t* l_cnt = reinterpret_cast<uint32_t*>(sl + kSlCnt);
    int32_t* l_S = reinterpret_cast<int32_t*>(sl + kSlS);
    int32_t* l_VI = reinterpret_cast<int32_t*>(sl + kSlVI);
    int32_t* l_BV = reinterpret_cast<int32_t*>(sl + kSlBV);
    int32_t* l_HI = l_BV + kWarp;  // list ends (the vectorised walk)
    int4* l_GE = reinterpret_cast<int4*>(sl + kSlS);  // the vectorised walk's layout of the same area
    uint32_t* l_bm = reinterpret_cast<uint32_t*>(sl + kSlBm);
    WarpQueue Q;
    Q.pos = reinterpret_cast<int32_t*>(sl + kSlQ);
    Q.vi = Q.pos + kQueue;
    Q.n = 0;
    // rows are taken from the top id down: the top quarter of the ids (the
    // rows whose out-neighbours have the longest lists) one row per turn, the
    // rest kVertexBatch rows per turn, so no warp is left with a long batch
    // while the others idle
    const int64_t t1 = (mine + 3) / 4;
    for (;;) {
        unsigned g = 0;
        if (lane == 0) g = atomicAdd(&s_light, 1u);
        const int64_t t = __shfl_sync(kFull, g, 0);
        const int64_t b = t < t1 ? t : t1 + (t - t1) * kVertexBatch;
        const int nq = t < t1 ? 1 : kVertexBatch;
        if (b >= mine) break;
        for (int q = 0; q < nq; q++) {
            const int64_t k = mine - 1 - (b + q);
            if (k < 0) break;
            const int64_t uu = first + k * step;
            const int32_t bu = G.begin(uu);
            const int d = (int)(G.end(uu) - bu);
            if (d < 2 || d > warp_cap) continue;
            RowState R = stage_row(G, A, l_su, l_cnt, l_bm, kLightBmLog2, true, bu, d, lane, kWarp, false);
            __syncwarp();
            const int vend = d;
            for (int vb = 0; vb < vend; vb += kWarp) {
                const int i = vb + (int)lane;
                int32_t len = 0;
                int32_t bv = 0;
                if (i < vend) {
                    const int32_t v = l_su[i];
                    if (v >= 0 && v < nv) {
                        bv = (int32_t)G.begin(v);
                        len = (int32_t)(G.end(v) - bv);
                    }
                }
                const int32_t units = kVec ? (len > 0 ? ((bv + len + 3) >> 2) - (bv >> 2) : 0) : len;
                const unsigned nem = __ballot_sync(kFull, len > 0);
                const int32_t incl = warp_incl_scan(units);
                const int total = __shfl_sync(kFull, incl, 31);
                if (len > 0) {
                    const int ci = __popc(nem & lanemask_lt());
                    if (kVec) {
                        l_GE[ci] = make_int4(incl - units, bv, bv + len, i);
                    } else {
                        l_S[ci] = incl - units;
                        l_VI[ci] = i;
                        l_BV[ci] = bv;
                        l_HI[ci] = bv + len;
                    }
                }
                __syncwarp();
                if (total > 0) {
                    if (kVec) walk_group_vec(G, A, R, l_GE, __popc(nem), 0, total, 0, Q);
                    else walk_group(G, A, R, l_S, l_VI, l_BV, __popc(nem), 0, total, 0, Q);
                }
                __syncwarp();
            }
            drain(G, A, R, Q);
            flush_row(R, A, lane, kWarp);
            __syncwarp();
        }
    }
}

// Drop-in support operator: accumulates into out; no scratch.
int launch_support_accum_i32(const int32_t* rp, int32_t stride, const int32_t* cols, int64_t nv, int64_t ne,
                             int32_t* out, cudaStream_t st) {
    if (nv <= 0) return TDT_OK;
    DeviceInfo di;
    int rc = device_info(&di);
    if (rc) return rc;
    OutRows G{rp, stride, cols, nv, ne};
    SupArgs A{};
    A.out = out;
    A.warp_cap = (g_warp_cap > 0 && g_warp_cap < kWarpCap) ? g_warp_cap : kWarpCap;
    A.heavy_cap = (g_heavy_cap > 0 && g_heavy_cap < kHeavyCap) ? g_heavy_cap : kHeavyCap;
    // the vectorised walk needs 16-byte aligned columns (chunk positions stay
    // below 2^31 under 2^30 edges)
    const bool vec = g_vec_walk && ((uintptr_t)cols & 15u) == 0 && ne < (1ll << 30);
    auto kern = vec ? support_kernel<true> : support_kernel<false>;
    TDT_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSupSmemBytes));
    TDT_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, 100));
    int blocks_per_sm = 0;
    TDT_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks_per_sm, kern, kSupBlock, kSupSmemBytes));
    if (blocks_per_sm < 1) blocks_per_sm = 1;
    kern<<<di.sms * blocks_per_sm, kSupBlock, kSupSmemBytes, st>>>(G, A);
    TDT_LAUNCH_CHECK("support");
    return TDT_OK;
}

}  // namespace tdt
