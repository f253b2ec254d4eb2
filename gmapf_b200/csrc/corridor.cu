// corridor.cu -- the search of search.cu (same rounds, same results) for maps of
// long corridors, where a search is thousands of rounds of a thin front.
//
// What bounds it: a search is a chain of dependent rounds, and a round a chain
// of dependent instructions with L2 reads in it.  On the 160x160-cell maze 95%
// of a search's rounds do not touch a queue: every claimed node is the next pop
// of the lane it goes to.  So this kernel makes that round short and gives the
// other rounds a slow path, where search.cu spends the same effort on both:
//   - edge rows (EdgeRow): a node together with the neighbour it was reached
//     from names its two other neighbours, their centroids and their own edge
//     rows: no neighbour list to sort out, no parent to leave out;
//   - one candidate per lane while at most 16 nodes expand (lane q and lane
//     q + 16 take the two candidates of node q): no compaction, no shuffles;
//   - each candidate's own edge row is copied into shared memory
//     (cp.async) while its visited state is checked: a round waits for one L2
//     access instead of two in a row;
//   - two candidates for one node are told apart by a hashed bit per candidate;
//     only rounds with a match compare nodes (search.cu: a MATCH.ANY over all
//     candidates of every round);
//   - claims go to a log in claim order (16 bytes, consecutive) instead of a
//     32-byte record per node scattered over the slot, half the DRAM writes,
//     and nothing is read back: an item's place in the log follows from its
//     place in the frontier;
//   - the queues move to global memory where that gives more resident warps
//     (they are rarely touched).
// Visited state: placement 1 (bitmap in shared memory) or 4 (bitmap in global
// memory, moved to shared memory at a batch's tail); see search.cu.
#include <cuda_runtime.h>

#include <mutex>
#include <type_traits>

#include "internal.h"
#include "records.cuh"
#include "region_plan.cuh"
#include "search_common.cuh"

namespace gmapf_b200 {

namespace {

// The claim log: entry i of a search is its i-th claim, {directed edge, G<<1|dir,
// parent's entry, jump ancestor's entry}; the jump ancestor is the nearest
// proper ancestor whose depth (G) is a multiple of kJumpDepth (-1: a root).
constexpr int kJumpDepth = 32;

// An entry as it is: one 16-byte access.
struct WideLog {
    int4* p;
    __device__ __forceinline__ WideLog(const SearchParams& a, int slot)
        : p(static_cast<int4*>(a.log) + (size_t)(a.slot_base + slot) * a.n) {}
    __device__ __forceinline__ int2 hop(int i) const {  // {directed edge, parent's entry}
        const int4 q = __ldcg(p + i);
        return make_int2(q.x, q.z);
    }
    __device__ __forceinline__ int edge(int i) const { return __ldcg(&p[i].x); }
    __device__ __forceinline__ int2 edge_jump(int i) const {
        const int4 q = __ldcg(p + i);
        return make_int2(q.x, q.w);
    }
    __device__ __forceinline__ int jump(int i) const { return __ldcg(&p[i].w); }
    __device__ __forceinline__ int depth(int i) const { return __ldcg(&p[i].y) >> 1; }
    __device__ __forceinline__ void put(int i, int e, int gd, int parent, int jump) const {
        __stcg(p + i, make_int4(e, gd, parent, jump));
    }
};

// The depth of an entry that does not keep it follows from the jump chain's length.
template <class LG>
__device__ __noinline__ int depth_by_jumps(LG log, int i) {
    const int first = log.jump(i);  // the nearest ancestor at a multiple of kJumpDepth
    if (first < 0) return 0;        // a root
    int d = 0;
    for (int x = i; x != first && x >= 0 && d <= kJumpDepth; x = log.hop(x).y) d++;
    for (int y = first; (y = log.jump(y)) >= 0;) d += kJumpDepth;  // (ever earlier entries)
    return d;
}

// In 8 bytes, for maps of at most 2^20 triangles: edge 22 bits, parent + 1 and
// jump + 1 20 bits each (an ancestor is an earlier claim).
struct HalfLog {
    unsigned long long* p;
    __device__ __forceinline__ HalfLog(const SearchParams& a, int slot)
        : p(static_cast<unsigned long long*>(a.log) + (size_t)slot * a.n) {}
    __device__ __forceinline__ unsigned long long at(int i) const { return __ldcg(p + i); }
    __device__ __forceinline__ int2 hop(int i) const {
        const unsigned long long v = at(i);
        return make_int2((int)(v & 0x3fffffu), (int)((v >> 22) & 0xfffffu) - 1);
    }
    __device__ __forceinline__ int edge(int i) const { return (int)(at(i) & 0x3fffffu); }
    __device__ __forceinline__ int jump(int i) const { return (int)(at(i) >> 42) - 1; }
    __device__ __forceinline__ int2 edge_jump(int i) const {
        const unsigned long long v = at(i);
        return make_int2((int)(v & 0x3fffffu), (int)(v >> 42) - 1);
    }
    __device__ __forceinline__ int depth(int i) const { return depth_by_jumps(*this, i); }
    __device__ __forceinline__ void put(int i, int e, int, int parent, int jump) const {
        __stcg(p + i, (unsigned long long)(unsigned)e | (unsigned long long)(unsigned)(parent + 1) << 22 |
                          (unsigned long long)(unsigned)(jump + 1) << 42);
    }
};
static_assert(kHalfLogNodes <= 1 << 20, "HalfLog: an edge has 22 bits, an entry 20");

// In 6 bytes, for maps of at most kPackedLogNodes triangles: a word of the edge (17
// bits) and parent + 1 (15; an ancestor is an earlier claim), a half word of
// jump + 1.  2.7 times the searches of WideLog in a fixed scratch array (searches
// without allocation).  Where memory is not the limit the wide entry costs fewer
// instructions: 64x64-cell maze, placement 1, against entries of 8 bytes, 16,384
// searches at T=4 14.5 to 14.9 ms, T=8 6.9 to 7.0, 37 searches 0.575 to 0.603; at
// T=32 the packed one was 0-6% faster, within what its runs differ by.
struct PackedLog {
    unsigned* p;         // slots x n words, then slots x n half words
    unsigned short* pj;
    __device__ __forceinline__ PackedLog(const SearchParams& a, int slot)
        : p(static_cast<unsigned*>(a.log) + (size_t)slot * a.n),
          pj(reinterpret_cast<unsigned short*>(static_cast<unsigned*>(a.log) + (size_t)a.slots * a.n) +
             (size_t)slot * a.n) {}
    __device__ __forceinline__ int2 hop(int i) const {
        const unsigned v = __ldcg(p + i);
        return make_int2((int)(v & 0x1ffffu), (int)(v >> 17) - 1);
    }
    __device__ __forceinline__ int edge(int i) const { return (int)(__ldcg(p + i) & 0x1ffffu); }
    __device__ __forceinline__ int jump(int i) const { return (int)__ldcg(pj + i) - 1; }
    __device__ __forceinline__ int2 edge_jump(int i) const { return make_int2(edge(i), jump(i)); }
    __device__ __forceinline__ int depth(int i) const { return depth_by_jumps(*this, i); }
    __device__ __forceinline__ void put(int i, int e, int, int parent, int jump) const {
        __stcg(p + i, (unsigned)e | (unsigned)(parent + 1) << 17);
        __stcg(pj + i, (unsigned short)(jump + 1));
    }
};
static_assert(kPackedLogNodes <= 1 << 15, "PackedLog: an edge has 17 bits, an entry 15");

// bounded push (CuQueue.h:33-63 with the (F,G,id) order) into a ring holding
// at most cap entries, kept in descending order (minimum at the tail)
// (entries keep their place in the claim log; their directed edge is read from
// there only to break a tie of F and G)
template <class LG>
__device__ __forceinline__ bool entry_less(LG log, int2 a, int ia, float F, int gd, int e, bool flip) {
    const float fa = __int_as_float(a.x);
    if (fa != F) return flip ? F < fa : fa < F;
    if ((a.y | 1) != (gd | 1)) return flip ? (gd | 1) < (a.y | 1) : (a.y | 1) < (gd | 1);
    const int ea = log.edge(ia);
    return flip ? e < ea : ea < e;
}

template <class LG>
__device__ __forceinline__ void ring_push(const Ring& r, LG log, int& beg, int& size, int cap, float F, int gd, int e,
                                          int id) {
    if (cap <= 0) return;
    if (size == cap) {
        const int k0 = r.at(beg);
        if (!entry_less(log, r.fg()[k0], r.id()[k0], F, gd, e, true))
            return;                            // not below the maximum: dropped
        beg = (beg + 1 == r.C) ? 0 : beg + 1;  // evict the maximum
        size--;
    }
    int i = size - 1;
    while (i >= 0) {
        const int k = r.at(beg + i);
        const int2 q = r.fg()[k];
        const int qi = r.id()[k];
        if (!entry_less(log, q, qi, F, gd, e, false)) break;
        const int k1 = r.at(beg + i + 1);
        r.fg()[k1] = q;
        r.id()[k1] = qi;
        i--;
    }
    const int k1 = r.at(beg + i + 1);
    r.fg()[k1] = make_int2(__float_as_int(F), gd);
    r.id()[k1] = id;
    size++;
}

// The round's frontier: 3T entries {F, G<<1|dir, directed edge, jump ancestor's
// log entry}; and a bit per hashed candidate of the round (4,096 bits: of 20
// candidates, 1 round in 20 has a false match, which costs one step of the loop
// over doubtful candidates).
constexpr int kSeenWords = 128;
// the edge rows of the round's candidates (the next round's starting points): one per lane, two in wide rounds
__host__ __device__ __forceinline__ constexpr int corridor_staged_rows(int T) { return T > 16 ? 64 : 32; }
__host__ __device__ __forceinline__ size_t corridor_frontier_words(int T) {
    return (size_t)4 * 3 * T + kSeenWords + 8 * corridor_staged_rows(T) + ((3 * T + 15) / 16) * 4;
}

// The log entry of node n (claimed by this search), newest first; -1 if none.  The other side's claim of the meeting node can be old (a queue
// dropped it): on the 160x160 maze 9-15 thousand claims back on average.
template <class LG>
__device__ __noinline__ int find_claim(LG log, int claims, int n, int lane) {
    constexpr int U = 8;  // 256 entries per step, all reads in flight
    for (int top = claims; top > 0; top -= 32 * U) {
        int q[U];
#pragma unroll
        for (int j = 0; j < U; j++) {
            const int i = top - 1 - (j * 32 + lane);
            q[j] = i >= 0 ? log.edge(i) : -1;
        }
        int hit = -1;
#pragma unroll
        for (int j = 0; j < U; j++)
            if ((q[j] >> 2) == n) hit = top - 1 - (j * 32 + lane);
        const unsigned m = __ballot_sync(kFull, hit >= 0);
        if (m) return __shfl_sync(kFull, hit, __ffs(m) - 1);
    }
    return -1;
}

// Path walk of one warp.  Lanes 0 and 1 follow each side's jump chain from the
// meeting pair and leave the checkpoints' log entries (the path nodes at depths
// that are multiples of kJumpDepth) at their output positions; then all lanes
// walk the segments between checkpoints, kJumpDepth hops each, and write the
// nodes.  A path of g hops per side takes about g / kJumpDepth + kJumpDepth
// dependent reads.
// A short search's log is read into shared memory (buf, cap entries) first and
// followed there.
template <class LG>
__device__ __forceinline__ void walk_path(LG log, int claims, int2* buf, int cap, int* out, int mS, int gS,
                                          int mT, int gT, int lane, int* err) {
    if (claims <= cap) {
        __syncwarp();
#pragma unroll 4
        for (int i = lane; i < claims; i += 32) {
            const int2 q = log.hop(i);
            buf[i] = make_int2(q.x >> 2, q.y);
        }
        __syncwarp();
        if (lane < 2) {
            int x = lane == 0 ? mS : mT;
            const int last = lane == 0 ? 1 : 0;
            for (int d = lane == 0 ? gS : gT; d >= last; d--) {
                if ((unsigned)x >= (unsigned)claims) {
                    atomicOr(err, ERR_BOUNDS);
                    break;
                }
                const int2 q = buf[x];
                out[path_pos(lane, d, gS, gT)] = q.x;
                x = q.y;
            }
        }
        return;
    }
    // checkpoints k*D, k = 1..K of each side: K = (g - 1) / D
    int kc = 0;
    bool bad = false;
    if (lane < 2) {
        const int g = lane == 0 ? gS : gT;
        int x = lane == 0 ? mS : mT;
        kc = g >= 1 ? (g - 1) / kJumpDepth : 0;
        for (int k = kc; k >= 1 && !bad; k--) {
            x = log.jump(x);  // the nearest ancestor at a multiple of D: depth k*D
            bad = x < 0 || x >= claims;
            if (!bad) out[path_pos(lane, k * kJumpDepth, gS, gT)] = x;
        }
    }
    const int kS = __shfl_sync(kFull, kc, 0), kT = __shfl_sync(kFull, kc, 1);
    const bool stop = __any_sync(kFull, bad);
    if (stop) {
        if (lane == 0) atomicOr(err, ERR_BOUNDS);
        return;
    }
    __syncwarp();  // the checkpoints are written
    // segment k of a side: k = 0 from the meeting node (its own node written
    // too) down to depth kD + 1 (or the side's last depth), k >= 1 from the
    // checkpoint at depth kD
    const int m = kS + 1 + kT + 1;
    constexpr int W = 4;  // segments per lane in flight: their reads do not wait for one another
    for (int i0 = lane; i0 < m; i0 += 32 * W) {
        int x[W], d[W], b[W], sd[W];
#pragma unroll
        for (int j = 0; j < W; j++) {
            const int i = i0 + 32 * j;
            x[j] = d[j] = b[j] = 0;
            sd[j] = 0;
            if (i < m) {
                const int side = i <= kS ? 0 : 1;
                const int k = side == 0 ? i : i - (kS + 1);
                const int kk = side == 0 ? kS : kT;
                const int last = side == 0 ? 1 : 0;
                sd[j] = side;
                if (k == 0) {
                    x[j] = side == 0 ? mS : mT;
                    d[j] = side == 0 ? gS : gT;
                    b[j] = kk >= 1 ? kk * kJumpDepth + 1 : last;
                } else {
                    d[j] = k * kJumpDepth;
                    x[j] = out[path_pos(side, d[j], gS, gT)];
                    b[j] = k == 1 ? last : (k - 1) * kJumpDepth + 1;
                }
            } else {
                d[j] = -1;
            }
        }
        bool more = true;
        while (more) {
            more = false;
            int2 q[W];
#pragma unroll
            for (int j = 0; j < W; j++) {
                if (d[j] < b[j]) continue;
                if (x[j] < 0 || x[j] >= claims) {
                    atomicOr(err, ERR_BOUNDS);
                    d[j] = -1;
                    b[j] = 0;
                    continue;
                }
                q[j] = log.hop(x[j]);
            }
#pragma unroll
            for (int j = 0; j < W; j++) {
                if (d[j] < b[j]) continue;
                out[path_pos(sd[j], d[j], gS, gT)] = q[j].x >> 2;
                x[j] = q[j].y;
                d[j]--;
                more = true;
            }
        }
    }
}

// per-block dynamic shared memory: per warp the queues (unless they are in
// global memory), the frontier and, in placement 1, the visited bitmap; in
// placement 4 a pad so that all but the first warp's share can hold one bitmap
// -- or, with full_pad, room for one whole bitmap: in a batch with a warp for
// every request, a search of each block moves its bitmap there while the
// block's others still run (2,047 searches, 160x160 maze: T=8 25.6 -> 24.1 ms,
// T=32 10.2 -> 9.4).  In larger batches it would be taken by whichever search
// comes first, not by the one that ends the batch (16,384 searches at T=32:
// 19.0 ms from the start on, 16.9 from the moment no request is left, 16.6 as
// search.cu does it, once the block's other warps have left).
size_t smem_bytes(int C, int bt, int bm_words, int T, int vm, bool queues_global, bool full_pad) {
    const size_t warps = (size_t)bt / 32;
    const size_t per_warp = (queues_global ? 0 : search_queue_words(C, T)) + corridor_frontier_words(T);
    const size_t pad = vm != 4 ? 0 : full_pad ? (size_t)bm_words : search_pad_words(bm_words, (int)warps, (int)per_warp);
    return 4 * (warps * (per_warp + (vm == 1 ? (size_t)bm_words : 0)) + pad);
}

// VM: visited placement (1 shared-memory bitmap, 4 global bitmap that a search
// still running at a batch's tail moves into the shared memory of its block's
// finished warps, as in search.cu).  A bit set by one thread is seen by the
// others after the next __syncwarp.
template <int T, int VM, class LG>
__global__ void __launch_bounds__(256, 3) k_corridor_search(SearchParams p, int persistent, int req_base, int bm_words) {
    constexpr bool SMEMV = VM == 1;  // bitmap in shared memory
    extern __shared__ __align__(16) unsigned char smem[];
    const int lane = threadIdx.x & 31;
    const int wib = threadIdx.x >> 5;                 // warp in block
    const int wpb = blockDim.x >> 5;                  // warps per block
    const int slot = blockIdx.x * wpb + wib;          // one request slot per warp
    const int n_nodes = p.n;
    const float K = p.K;
    const int C = p.C;
    // placement 4: the warps of this block that have left the persistent loop
    // (or never entered it; their shares stay free) and the warp whose search
    // runs in the block's shared memory (-1: none)
    __shared__ unsigned block_left;
    __shared__ int block_mover;
    if constexpr (VM == 4) {
        if (threadIdx.x == 0) {
            const int valid = max(0, min(wpb, p.slots - (int)blockIdx.x * wpb));
            block_left = (wpb >= 32 ? 0xffffffffu : ((1u << wpb) - 1u)) & ~((valid >= 32 ? 0xffffffffu : (1u << valid) - 1u));
            block_mover = -1;
        }
        __syncthreads();
    }

    // shared memory: [queues of every warp][frontiers of every warp][bitmaps]
    // (placement 4: [queues | frontier] of each warp, then the pad), each
    // per-warp region a whole number of 16-byte words
    // (the queues are in global memory when p.queues is set)
    const size_t qwords = search_queue_words(C, T);
    const size_t qblk = p.queues ? 0 : qwords, fblk = corridor_frontier_words(T);
    int* base = reinterpret_cast<int*>(smem);
    Ring ring;
    int* share = VM == 4 ? base + (size_t)wib * (qblk + fblk) : base + (size_t)wib * qblk;
    ring.base = p.queues ? p.queues + (size_t)(p.slot_base + slot) * qwords : share;
    ring.T = T;
    ring.q = lane & (T - 1);  // (lanes >= T own no queue)
    ring.C = C;
    int4* fr = reinterpret_cast<int4*>(VM == 4 ? share + qblk : base + (size_t)wpb * qblk + (size_t)wib * fblk);
    unsigned* bm = SMEMV ? reinterpret_cast<unsigned*>(base + (size_t)wpb * (qblk + fblk)) + (size_t)wib * bm_words
                         : nullptr;

    if (slot >= p.slots) return;  // whole warps
    if (VM == 4) bm = p.gbm + (size_t)(p.slot_base + slot) * bm_words;
    const LG log(p, slot);
    const unsigned lt_mask = (1u << lane) - 1u;

    for (int iter = 0;; iter++) {
        // ------------------------------------------------------------ fetch
        int r, R;
        bool queue_feeds = false;  // warps come back for more requests
        if (persistent) {
            R = p.starts ? p.req_count_h : *p.req_count_d;
            // a batch with a warp for every request: warp 0 of every block first, so
            // that it spreads over the SMs, and no warp asks the counter
            const int warps = (int)gridDim.x * wpb;
            queue_feeds = !(R <= warps && warps <= p.slots);
            if (!queue_feeds) {
                r = iter == 0 ? wib * (int)gridDim.x + (int)blockIdx.x : R;
            } else {
                int v = 0;
                if (lane == 0) v = atomicAdd(p.work_ctr, 1);
                r = __shfl_sync(kFull, v, 0);
            }
        } else {
            if (iter > 0) break;
            r = req_base + slot;
            R = p.req_count_h;
        }
        if (r >= R) break;
        // ring entries are rewritten by host copies over time: read past L1
        const int4 rq = p.starts         ? make_int4(-1, p.starts[r], p.targets[r], r)
                        : p.ring_cap > 0 ? __ldcg(p.req + ((p.ring_base + r) % p.ring_cap)) : p.req[r];
        const int agent = rq.x, start = rq.y, target = rq.z, orow = rq.w;
        if (start < 0 || start >= n_nodes || target < 0 || target >= n_nodes || start == target) {
            const bool bad = start != target || start < 0 || start >= n_nodes;
            if (lane == 0) {  // bad request: not found; start == target: found, empty path
                if (p.timeline) p.timeline[2 * (long long)orow] = p.timeline[2 * (long long)orow + 1] = global_timer_ns();
                if (bad) atomicOr(p.err, ERR_BAD_REQUEST);
                if (p.out_found) p.out_found[orow] = bad ? p.bad_code : 1;
                if (p.out_len) p.out_len[orow] = 0;
                if (agent >= 0 && p.ag_state) {
                    p.ag_state[agent] = GMAPF_AGENT_IDLE;
                    p.ag_path_len[agent] = 0;
                }
                if (!bad && p.stats) atomicAdd(p.stats + ST_FOUND, 1ull);
                if (p.done) ring_complete(p, orow, p.ring_base + r, bad ? 0 : 1);
            }
            continue;
        }

        if (p.timeline && lane == 0) p.timeline[2 * (long long)orow] = global_timer_ns();
        uint4* b4 = reinterpret_cast<uint4*>(bm);
        for (int k = lane; k < (bm_words >> 2); k += 32) {
            if (SMEMV) b4[k] = make_uint4(0, 0, 0, 0);
            else __stcg(b4 + k, make_uint4(0, 0, 0, 0));
        }
        __syncwarp();
        const float2 cs = p.cen[start];
        const float2 ct = p.cen[target];
        // Queue q is kept by lane q (and, while T <= 16, mirrored by lane q + 16):
        // the node selected for the coming round -- its directed edge e (node << 2
        // | slot of its parent, -1 if none), its place in the claim log and its
        // jump ancestor's -- and the ring in shared memory with its minimum cached
        // in registers (t*).
        //
        // Candidates per lane: with at most 16 nodes to expand (always for
        // T <= 16, in most rounds of T = 32), lane q takes the first candidate of
        // node q and lane q + 16 the second (a narrow round: one candidate per
        // lane, half the instructions); else lane q takes both.
        constexpr bool MIRROR = T <= 16;
        bool narrow = true;
        bool staged = false;  // the frontier items' edge rows are beside them
        int qbeg = 0, qsize = 0;
        struct Key {
            float F;
            int gd, e, at, jump;
        };
        Key top{0.f, 0, -1, 0, -1};  // the ring's minimum
        int e = -1, gd = 0, at = 0, jump = -1;
        EdgeHalf c0, c1;  // the lane's candidates (c1: wide rounds only)
        auto load_selected = [&]() {
            if (MIRROR || narrow)
                ld_edge_half(&p.erow->x, e < 0 ? -1 : 2 * (long long)e + (lane >> 4), c0);
            else
                ld_edge_row(p.erow, e, c0, c1);
        };
        // Lanes 0 and 1 seed the start and the target (PathFinder.h:168-189); a
        // root may have three candidates: the first round takes the third on
        // lanes 8 and 9.
        if ((lane & 7) < 2 && lane != 24 && lane != 25) {
            const int k = lane & 7;
            const int node = k == 0 ? start : target;
            gd = k == 0 ? 1 : 0;
            e = (node << 2) | 3;
            at = k;
            if (lane < 2) {
                log.put(lane, e, gd, -1, -1);
                bm_set<SMEMV>(bm, node, gd);
            }
        }
        // (a seed's F never takes part in a comparison: each seed is alone in its queue)
        reinterpret_cast<int4*>(fr + 3 * T)[lane] = make_int4(0, 0, 0, 0);
        __syncwarp();
        load_selected();
        if ((lane & 15) == 8 || (lane & 15) == 9) ld_edge_half(p.third, e < 0 ? -1 : e >> 2, c0);
        // A root's third candidate is in its slot 2, as is one of the other root's when
        // ids outside the navmesh leave a slot empty: by lane, the start's would come
        // after the target's.  Such a candidate is in the second half, marked
        // (noalloc.cu), and the first round goes pass by pass.
        if (lane < 2) c0.info &= ~kEdgeThird;

        unsigned deg_sum = 0;
        int rounds = 0, expansions = 0, active = 2;  // active: nodes expanded by the coming round
        int claims = 2;                              // = entries of the claim log
        bool cut = false;  // stopped by the round limit
        int found = 0, mS = -1, gS = 0, mT = -1, gT = 0;  // the meeting pair: log entries and depths
        int next_check = p.promote_rounds;  // placement 4: the round of the next room-in-block check

        // ------------------------------------------------------------ rounds
        // The rounds with the claim checks in placement VX (1 shared, 3 global
        // bitmap) on bitmap bmx.  Returns true when the
        // search has ended, false when (placement 4) enough warps of its block
        // have left for its bitmap to fit in their shares.
        auto run_rounds = [&](auto vtag, unsigned* bmx) -> bool {
          constexpr int VX = decltype(vtag)::value;
          constexpr bool SMX = VX == 1;
          // a hashed bit of the round: candidates for one node take the same one
          unsigned* seen = reinterpret_cast<unsigned*>(fr + 3 * T);
          // the edge row of each candidate, and of frontier item i which it is
          EdgeHalf* rows = reinterpret_cast<EdgeHalf*>(fr + 3 * T + kSeenWords / 4);
          unsigned char* row_at = reinterpret_cast<unsigned char*>(rows + 2 * corridor_staged_rows(T));
          auto visited = [&](int n) -> int { return SMX ? bm_get(bmx, n) : bm_bits(__ldcg(bmx + (n >> 4)), n); };
          auto set_visited = [&](int n, int dir) { bm_set<SMX>(bmx, n, dir); };
          // One round's claims: writes its frontier, returns the number of claims, or
          // -1 when the two sides met (or an index check failed).
          auto claim_round = [&](auto ntag) -> int {
            constexpr int NC = decltype(ntag)::value;  // candidates per lane: 1 narrow, 2 wide
            const int du = gd & 1, ngd = gd + 2;  // the candidates' side and (G + 1) << 1 | side
            const float gf = (float)(ngd >> 1), farx = du ? ct.x : cs.x, fary = du ? ct.y : cs.y;
            // the children's jump ancestor: this node when its depth is a multiple of kJumpDepth, else its own
            const int cjump = ((gd >> 1) & (kJumpDepth - 1)) == 0 ? at : jump;
            // a claim: frontier entry i of the round = log entry claims + i
            auto write_claim = [&](int i, int en, float cx, float cy) {
                const float F = GM_FADD(gf, GM_FMUL(dist_sqr(cx, cy, farx, fary), K));
                fr[i] = make_int4(__float_as_int(F), ngd, en, cjump);
                log.put(claims + i, en, ngd, at, cjump);
            };

            // the search's end: node mn, log entry `other` (-1: look for it), met from log entry mat with key mgd
            auto finish = [&](int mat, int mgd, int mn, int other) {
                if (other < 0) other = find_claim(log, claims, mn, lane);
                if (other < 0) {
                    if (lane == 0) atomicOr(p.err, ERR_BOUNDS);
                    return;
                }
                const int og = log.depth(other);
                const bool from_start = mgd & 1;  // PathFinder.h:226-227
                mS = from_start ? mat : other;
                gS = from_start ? mgd >> 1 : og;
                mT = from_start ? other : mat;
                gT = from_start ? og : mgd >> 1;
                found = 1;
            };
            // A candidate whose node nobody claimed is this lane's claim (g) unless
            // another lane of the round asks for the same node (s).
            EdgeHalf c[NC];
            int n[NC];
            bool g[NC], s[NC];
            const bool odd = (c0.info & kEdgeThird) != 0;  // a third candidate
            bool doubt = odd;
            bool cross[NC];  // claimed earlier from the other side: the sides meet
#pragma unroll
            for (int j = 0; j < NC; j++) {
                c[j] = j == 0 ? c0 : c1;
                n[j] = max(c[j].e, 0) >> 2;
                g[j] = c[j].e >= 0;
                // the candidate's own edge row, for the round that expands it
                copy_edge_row(rows + 2 * (j * 32 + lane), p.erow, c[j].e);
                // (lanes without a candidate set no bit, each in its own word: no branch)
                const unsigned bit = g[j] ? 1u << (n[j] & 31) : 0u;
                const unsigned taken = atomicOr(seen + (g[j] ? (n[j] >> 5) & (kSeenWords - 1) : lane), bit) & bit;
                const int v = SMX ? (g[j] ? bm_get(bmx, n[j]) : 0) : bm_bits(ld_word_if(bmx + (n[j] >> 4), g[j]), n[j]);
                cross[j] = v != 0 && (v >> 1) != du;
                g[j] = g[j] && v == 0;
                s[j] = g[j] && taken;
                g[j] = g[j] && !taken;
                doubt = doubt || s[j] || cross[j];
            }
            int meet_key = 0x7fffffff;  // (slot, queue) of the first candidate claimed earlier from the other side
            if (__any_sync(kFull, doubt)) {
                bool passes = __any_sync(kFull, odd);
                if (!passes) {
                    // (slot, queue) order, with the side in bit 0
                    int key[NC];
                    int mk = 0x7fffffff;
#pragma unroll
                    for (int j = 0; j < NC; j++) {
                        key[j] = (int)((c[j].info & 7u) << 6) | (NC > 1 ? lane : lane & 15) << 1 | du;
                        if (cross[j]) mk = min(mk, key[j]);
                    }
                    // Candidates for a node that another lane of the round holds, one
                    // by one: the first of them in candidate order (slot-major) keeps it.
#pragma unroll
                    for (int j = 0; j < NC; j++) {
                        for (unsigned m = __ballot_sync(kFull, s[j]); m && !passes; m &= m - 1) {
                            const int l = __ffs(m) - 1;
                            const int nl = __shfl_sync(kFull, n[j], l);
                            const unsigned h0 = __ballot_sync(kFull, g[0] && n[0] == nl);
                            const unsigned h1 = NC > 1 ? __ballot_sync(kFull, g[NC - 1] && n[NC - 1] == nl) : 0u;
                            if ((h0 | h1) == 0u) {
                                if (lane == l) g[j] = true;  // only its hashed bit was taken
                                continue;
                            }
                            const int h = __ffs(h0 ? h0 : h1) - 1;
                            const int kl = __shfl_sync(kFull, key[j], l);
                            const int kh = __shfl_sync(kFull, h0 ? key[0] : key[NC - 1], h);
                            if ((kl ^ kh) & 1) {
                                passes = true;  // the two sides meet in this round's claims
                            } else if (kl < kh) {
                                if (lane == h) (h0 ? g[0] : g[NC - 1]) = false;
                                if (lane == l) g[j] = true;
                            }
                        }
                    }
                    if (!passes) meet_key = __reduce_min_sync(kFull, mk);
                    if (meet_key != 0x7fffffff) {  // the sides meet: no need to place this round's claims
                        int nwin = 0, mn = 0;
                        unsigned who = 0;
#pragma unroll
                        for (int j = 0; j < NC; j++) {
                            nwin += __popc(__ballot_sync(kFull, g[j]));
                            const unsigned w = __ballot_sync(kFull, cross[j] && key[j] == meet_key);
                            if (w) {
                                who = w;
                                mn = __shfl_sync(kFull, n[j], __ffs(w) - 1);
                            }
                        }
                        const int ml = __ffs(who) - 1;
                        finish(__shfl_sync(kFull, at, ml), __shfl_sync(kFull, gd, ml), mn, -1);
                        claims += nwin;
                        return -1;
                    }
                }
                if (passes) {
                    // Pass by pass (neighbour slot 0 of every queue, then 1, then 2), in
                    // candidate order by thread: visited state, the lowest fresh
                    // thread of a node claims it, the first conflicting thread is
                    // the meeting pair.
                    // lane q gets all candidates of queue q
                    EdgeHalf x = c[0], y = c[NC - 1];
                    if (NC == 1) {
                        y.e = __shfl_sync(kFull, c[0].e, lane | 16);
                        y.info = __shfl_sync(kFull, c[0].info, lane | 16);
                        if (lane >= (rounds == 1 ? 2 : 16)) x.e = y.e = -1;
                    }
                    int ez = -1;
                    unsigned oz = 0;
                    if (x.e >= 0 && ((x.info & kEdgeThird) || rounds == 1)) {
                        ez = p.third[e >> 2].e;
                        oz = ~(x.info | y.info) & 7u;  // its slot is the one left
                    }
                    int nwin = 0, mat = 0, mgd = 0, mn = 0, other = -1;  // the pair: log entry, key; the node met, its log entry
                    bool meet = false;
#pragma unroll 1
                    for (unsigned one = 1; one < 8; one <<= 1) {
                        const int en = (x.e >= 0 && (x.info & one)) ? x.e : (y.e >= 0 && (y.info & one)) ? y.e : (oz & one) ? ez : -1;
                        const int nn = en >> 2;
                        const int st = en >= 0 ? visited(nn) : 0;  // (with the claims of earlier passes)
                        const bool fresh = en >= 0 && st == 0;
                        const unsigned dm = __ballot_sync(kFull, du);  // candidates' sides
                        const unsigned mm = __match_any_sync(kFull, fresh ? nn : -1);
                        const int leader = __ffs(mm) - 1;
                        const bool win = fresh && leader == lane;
                        const bool dup = fresh && !win;  // same node as a lower candidate of this pass
                        const bool conflict = dup ? (int)((dm >> leader) & 1u) != du : (en >= 0 && st && (st >> 1) != du);
                        const unsigned cm = __ballot_sync(kFull, conflict);
                        const unsigned wm = __ballot_sync(kFull, win);
                        if (!meet && cm != 0u) {  // warp-uniform
                            const int ml = __ffs(cm) - 1;
                            mat = __shfl_sync(kFull, at, ml);
                            mgd = __shfl_sync(kFull, gd, ml);
                            mn = __shfl_sync(kFull, nn, ml);
                            const int lead = __shfl_sync(kFull, dup ? leader : -1, ml);
                            if (lead >= 0) other = claims + nwin + __popc(wm & ((1u << lead) - 1u));
                            meet = true;
                        }
                        if (win) {
                            const float2 cn = p.cen[nn];
                            write_claim(nwin + __popc(wm & lt_mask), en, cn.x, cn.y);
                            set_visited(nn, du);
                        }
                        nwin += __popc(wm);
                        __syncwarp();
                    }
                    if (!meet) {
                        staged = false;
                        return nwin;
                    }
                    claims += nwin;
                    finish(mat, mgd, mn, other);
                    return -1;
                }
            }
            // candidate order: slot-major, queues ascending
            if constexpr (NC == 1) {
                const unsigned w = g[0] ? c[0].info : 0u;
                unsigned b0 = __ballot_sync(kFull, w & 1u), b1 = __ballot_sync(kFull, w & 2u), b2 = __ballot_sync(kFull, w & 4u);
                // (a queue has one candidate per slot, in either half)
                const unsigned b01 = ((b0 | b0 >> 16) & 0xffffu) | (b1 | b1 << 16) & 0xffff0000u;
                b2 = (b2 | b2 >> 16) & 0xffffu;
                const int n01 = __popc(b01);
                if (g[0]) {
                    const unsigned lt = (1u << (lane & 15)) - 1u;
                    const bool two = (w & 4u) != 0;
                    const int i = (two ? n01 : 0) + __popc((two ? b2 : b01) & ((w & 2u) ? lt << 16 | 0xffffu : lt));
                    write_claim(i, c[0].e, c[0].x, c[0].y);
                    set_visited(n[0], du);
                    row_at[i] = (unsigned char)lane;
                }
                return n01 + __popc(b2);
            } else {
                const unsigned w0 = g[0] ? c[0].info : 0u, w1 = g[1] ? c[1].info : 0u;
                const unsigned b0 = __ballot_sync(kFull, (w0 | w1) & 1u), b1 = __ballot_sync(kFull, (w0 | w1) & 2u),
                               b2 = __ballot_sync(kFull, (w0 | w1) & 4u);
                const int n0 = __popc(b0), n01 = n0 + __popc(b1);
#pragma unroll
                for (int j = 0; j < 2; j++) {
                    const unsigned w = j == 0 ? w0 : w1;
                    if (g[j]) {
                        const unsigned b = (w & 1u) ? b0 : (w & 2u) ? b1 : b2;
                        const int i = ((w & 1u) ? 0 : (w & 2u) ? n0 : n01) + __popc(b & lt_mask);
                        write_claim(i, c[j].e, c[j].x, c[j].y);
                        set_visited(n[j], du);
                        row_at[i] = (unsigned char)(j * 32 + lane);
                    }
                }
                return n01 + __popc(b2);
            }
          };
          for (;;) {
            rounds++;
            expansions += active;
            deg_sum += c0.info >> 4;
            int nwin;
            staged = true;
            if constexpr (MIRROR)
                nwin = claim_round(std::integral_constant<int, 1>{});
            else
                nwin = narrow ? claim_round(std::integral_constant<int, 1>{}) : claim_round(std::integral_constant<int, 2>{});
            copies_done();
            if (nwin < 0) return true;  // met
            __syncwarp();  // the frontier is written

            // ---- next pops.  Frontier item i goes to queue i mod T; pushing a
            // round's items and then popping the minimum equals selecting the
            // minimum of (ring + items) first and inserting the rest with
            // capacity C - 1.  In most rounds every queue gets at most one item and
            // none has a queued entry below it: the items are the next pops.
            const bool small = nwin <= 16;
            const int src = MIRROR || small ? lane & 15 : lane;
            const bool got = src < T && src < nwin;
            const int4 it = fr[src < 3 * T ? src : 0];
            const bool queued = qsize > 0;  // (0 on lanes that own no queue)
            // (a lane >= 16 has another lane's item while there are at most 16)
            const bool keep = queued && !(src == lane && got && key_less(__int_as_float(it.x), it.y, it.z, top.F, top.gd, top.e));
            if (nwin <= T && !__any_sync(kFull, keep)) {
                if (nwin == 0) return true;  // every queue is empty
                active = nwin;
                narrow = small;
                e = got ? it.z : -1;
                gd = it.y;
                at = claims + src;
                jump = it.w;
                if (staged) {  // the next pops' candidates are beside the frontier
                    const EdgeHalf* r = rows + 2 * row_at[got ? src : 0];
                    c0 = r[MIRROR || narrow ? lane >> 4 : 0];
                    if (!MIRROR) c1 = r[1];
                    if (!got) {
                        c0.e = c1.e = -1;
                        c0.info = 0;
                    }
                } else {
                    load_selected();
                }
            } else {
                // selects instead of a branch per received item (an absent item
                // reads entry 0 and is ignored)
                int pick = -1;
                bool have = queued;
                Key best = top;
                auto take = [&](int j) {
                    const int i = lane + j * T;
                    const bool there = lane < T && i < nwin;
                    const int4 x = fr[there ? i : 0];
                    const bool better = there && (!have || key_less(__int_as_float(x.x), x.y, x.z, best.F, best.gd, best.e));
                    pick = better ? i : pick;
                    have = have || better;
                    best.F = better ? __int_as_float(x.x) : best.F;
                    best.gd = better ? x.y : best.gd;
                    best.e = better ? x.z : best.e;
                    best.jump = better ? x.w : best.jump;
                };
                take(0);
                if (nwin > T) {
                    take(1);
                    take(2);
                }
                e = have ? best.e : -1;
                gd = best.gd;
                at = pick < 0 ? top.at : claims + pick;
                jump = best.jump;
                const bool pop_top = have && pick < 0;
                int rs = pick >= 0 && staged ? (int)row_at[pick] : -1;  // its edge row beside the frontier
                const int mine = pick;
                active = __popc(__ballot_sync(kFull, have));
                if (active == 0) return true;
                narrow = MIRROR;
                if (MIRROR) {
                    e = __shfl_sync(kFull, e, lane & 15);
                    gd = __shfl_sync(kFull, gd, lane & 15);
                    at = __shfl_sync(kFull, at, lane & 15);
                    jump = __shfl_sync(kFull, jump, lane & 15);
                    rs = __shfl_sync(kFull, rs, lane & 15);
                }
                if (rs >= 0) {
                    c0 = rows[2 * rs + (MIRROR ? lane >> 4 : 0)];
                    if (!MIRROR) c1 = rows[2 * rs + 1];
                } else {
                    load_selected();  // in flight during the insertions
                }
                if (lane < T) {
                    bool touched = pop_top;
                    if (pop_top) qsize--;
                    auto put = [&](int j) {
                        const int i = lane + j * T;
                        if (i < nwin && i != mine) {
                            const int4 x = fr[i];
                            ring_push(ring, log, qbeg, qsize, C - 1, __int_as_float(x.x), x.y, x.z, claims + i);
                            touched = true;
                        }
                    };
                    put(0);
                    if (nwin > T) {
                        put(1);
                        put(2);
                    }
                    if (touched && qsize > 0) {  // an untouched ring keeps its cached minimum
                        const int k = ring.at(qbeg + qsize - 1);
                        const int2 w = ring.fg()[k];
                        top.F = __int_as_float(w.x);
                        top.gd = w.y;
                        top.at = ring.id()[k];
                        const int2 c = log.edge_jump(top.at);
                        top.e = c.x;
                        top.jump = c.y;
                    }
                }
            }
            claims += nwin;
            if (rounds >= p.max_rounds) {  // still running after its last allowed round
                if (lane == 0) atomicOr(p.err, ERR_ROUNDS);
                cut = true;
                return true;
            }
            reinterpret_cast<int4*>(seen)[lane] = make_int4(0, 0, 0, 0);
            __syncwarp();  // frontier reads done before the next round rewrites it
            if constexpr (VM == 4 && VX == 3) {
                // at promote_rounds rounds, then every 256: enough shares free
                // (their count; where the bitmap goes is worked out outside)?
                if (rounds == next_check) {  // warp-uniform
                    next_check += 256;
                    int room = 0;
                    if (lane == 0)
                        room = p.full_pad && !queue_feeds
                                   ? *reinterpret_cast<volatile int*>(&block_mover) < 0
                                   : __popc(*reinterpret_cast<volatile unsigned*>(&block_left) | (1u << wib)) >=
                                         region_shares_needed(bm_words, wpb, (int)(qblk + fblk));
                    if (__shfl_sync(kFull, room, 0)) return false;
                }
            }
          }
        };
        if constexpr (VM == 4) {
            int move_plan = -1;
            while (!run_rounds(std::integral_constant<int, 3>{}, bm)) {
                if (lane == 0) {
                    move_plan = region_plan(*reinterpret_cast<volatile unsigned*>(&block_left), wib, wpb,
                                            (int)(qblk + fblk), bm_words,
                                            p.full_pad ? bm_words
                                                       : (int)search_pad_words(bm_words, wpb, (int)(qblk + fblk)));
                    if (move_plan >= 0 && atomicCAS(&block_mover, -1, wib) != -1) move_plan = -1;
                }
                move_plan = __shfl_sync(kFull, move_plan, 0);
                if (move_plan >= 0) break;  // else back to the rounds: the next check in 256
            }
            if (move_plan >= 0) {
                // shares of warps that have left hold the bitmap from share
                // `first` on; this warp's queues and frontier move to share `home`
                // when its own share lies in that run; the search goes on there
                __threadfence_block();
                const int first = move_plan & 0xff, home = move_plan >> 8;
                if (home != wib) {
                    const int4* from = reinterpret_cast<const int4*>(share);
                    int4* to = reinterpret_cast<int4*>(base + (size_t)home * (qblk + fblk));
                    for (int k = lane; k < (int)((qblk + fblk) >> 2); k += 32) to[k] = from[k];
                    __syncwarp();
                    int* there = base + (size_t)home * (qblk + fblk);
                    if (!p.queues) ring.base = there;
                    fr = reinterpret_cast<int4*>(there + qblk);
                }
                unsigned* region = reinterpret_cast<unsigned*>(base + (size_t)first * (qblk + fblk));
                const uint4* g4 = reinterpret_cast<const uint4*>(bm);
                uint4* s4 = reinterpret_cast<uint4*>(region);
                for (int k = lane; k < (bm_words >> 2); k += 32) s4[k] = __ldcg(g4 + k);
                __syncwarp();
                run_rounds(std::integral_constant<int, 1>{}, region);
                // back to the warp's own share (the next query starts afresh) and
                // the block's shared memory free for another search
                if (!p.queues) ring.base = share;
                fr = reinterpret_cast<int4*>(share + qblk);
                __syncwarp();
                __threadfence_block();
                if (lane == 0) {
                    atomicExch(&block_mover, -1);
                    atomicAdd(p.stats + ST_PROMOTED, 1ull);
                }
            }
        } else {
            run_rounds(std::integral_constant<int, VM>{}, bm);
        }

        // ------------------------------------------------------------ path walk
        int L = 0;
        if (found) {
            L = gS + gT + 1;
            const int row = (agent >= 0) ? agent : orow;
            if ((long long)L > p.path_stride) {
                if (lane == 0) atomicOr(p.err, ERR_PATH_CAP);
            } else {
                walk_path(log, claims, reinterpret_cast<int2*>(qblk > fblk ? share : reinterpret_cast<int*>(fr)),
                          (int)max(qblk, fblk) / 2, p.paths + (long long)row * p.path_stride, mS, gS, mT, gT, lane, p.err);
            }
        }
        __syncwarp();
        // results, agent update (PathFinder.h:268-289) and counters
        const unsigned ds = __reduce_add_sync(kFull, deg_sum);
        if (lane == 0) {
            if (p.out_found) p.out_found[orow] = cut ? p.cut_code : found;
            if (p.out_len) p.out_len[orow] = L;
            if (agent >= 0 && p.ag_state) {
                // PathFinder.h:268-289: not found -> Idle with the path step
                // index left as it was; found -> Move from step -1
                p.ag_state[agent] = found ? GMAPF_AGENT_MOVE : GMAPF_AGENT_IDLE;
                if (found) p.ag_step_idx[agent] = -1;
                p.ag_path_len[agent] = L;
            }
            if (p.stats) {
                atomicAdd(p.stats + ST_EXPANSIONS, (unsigned long long)expansions);
                atomicAdd(p.stats + ST_DEG_SUM, (unsigned long long)ds);
                atomicAdd(p.stats + ST_ROUNDS, (unsigned long long)rounds);
                atomicAdd(p.stats + ST_CLAIMS, (unsigned long long)claims);
                atomicAdd(p.stats + ST_PATH_NODES, (unsigned long long)L);
                atomicAdd(p.stats + ST_FOUND, (unsigned long long)found);
            }
            if (p.done) ring_complete(p, orow, p.ring_base + r, found);
            if (p.timeline) p.timeline[2 * (long long)orow + 1] = global_timer_ns();
        }
    }
    if constexpr (VM == 4) {  // this warp uses its block's shared memory no more
        __syncwarp();
        __threadfence_block();
        if (lane == 0) atomicOr(&block_left, 1u << wib);
    }
}

template <int T, int VM, class LG>
cudaError_t launch_t(cudaStream_t s, const SearchParams& p, int blocks, int bt, bool persistent,
                     int req_base, int bm_words) {
    // the dynamic shared-memory limit was raised when the search state was
    // sized (no attribute calls here: this may run under stream capture)
    const size_t smem = smem_bytes(p.C, bt, bm_words, T, VM, p.queues != nullptr, p.full_pad != 0);
    if (blocks <= 0) return cudaSuccess;
    k_corridor_search<T, VM, LG><<<blocks, bt, smem, s>>>(p, persistent ? 1 : 0, req_base, bm_words);
    return cudaGetLastError();
}

// the kernel's dynamic shared-memory limit (only ever raised, as for search.cu's kernel)
std::mutex g_smem_attr_mu;

template <int T, int VM, class LG>
bool raise_smem_limit(int smem) {
    static int limit[64] = {};
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    std::lock_guard<std::mutex> lock(g_smem_attr_mu);
    if (smem > limit[device & 63]) {
        if (cudaFuncSetAttribute(k_corridor_search<T, VM, LG>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) !=
            cudaSuccess) {
            cudaGetLastError();
            return false;
        }
        limit[device & 63] = smem;
    }
    return true;
}

template <int T, int VM, class LG>
int occupancy_t(int C, int bt, int bm_words, bool queues_global, bool full_pad) {
    if (bt > 256) return 0;  // the kernel's launch bounds
    const size_t smem = smem_bytes(C, bt, bm_words, T, VM, queues_global, full_pad);
    if (smem > 227 * 1024 || !raise_smem_limit<T, VM, LG>((int)smem)) return 0;
    int nb = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_corridor_search<T, VM, LG>, bt, smem) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return nb;
}

template <int VM, class LG>
cudaError_t launch_v(cudaStream_t s, const SearchParams& p, int blocks, int bt, bool persistent,
                     int req_base, int bm_words) {
    switch (p.T) {
        case 2: return launch_t<2, VM, LG>(s, p, blocks, bt, persistent, req_base, bm_words);
        case 4: return launch_t<4, VM, LG>(s, p, blocks, bt, persistent, req_base, bm_words);
        case 8: return launch_t<8, VM, LG>(s, p, blocks, bt, persistent, req_base, bm_words);
        case 16: return launch_t<16, VM, LG>(s, p, blocks, bt, persistent, req_base, bm_words);
        case 32: return launch_t<32, VM, LG>(s, p, blocks, bt, persistent, req_base, bm_words);
        default: return cudaErrorInvalidValue;
    }
}

template <int VM>
int occupancy_v(int T, int C, int bt, int bm_words, bool qg, bool full_pad) {
    switch (T) {
        case 2: return occupancy_t<2, VM, WideLog>(C, bt, bm_words, qg, full_pad);
        case 4: return occupancy_t<4, VM, WideLog>(C, bt, bm_words, qg, full_pad);
        case 8: return occupancy_t<8, VM, WideLog>(C, bt, bm_words, qg, full_pad);
        case 16: return occupancy_t<16, VM, WideLog>(C, bt, bm_words, qg, full_pad);
        case 32: return occupancy_t<32, VM, WideLog>(C, bt, bm_words, qg, full_pad);
        default: return 0;
    }
}

}  // namespace

size_t corridor_smem_bytes(int C, int bt, int bm_words, int T, int vm) {
    return smem_bytes(C, bt, bm_words, T, vm, false, false);
}

template <int T>
static bool full_smem_t() {
    constexpr int kAll = 227 * 1024;
    return raise_smem_limit<T, 1, WideLog>(kAll) && raise_smem_limit<T, 1, HalfLog>(kAll) &&
           raise_smem_limit<T, 1, PackedLog>(kAll);
}

bool corridor_full_smem(int T) {
    switch (T) {
        case 2: return full_smem_t<2>();
        case 4: return full_smem_t<4>();
        case 8: return full_smem_t<8>();
        case 16: return full_smem_t<16>();
        case 32: return full_smem_t<32>();
        default: return false;
    }
}

size_t corridor_queue_bytes(int C, int T) { return 4 * search_queue_words(C, T); }

int corridor_max_blocks_per_sm(int T, int C, int bt, int vm, int bm_words, bool queues_global, bool full_pad) {
    switch (vm) {
        case 1: return occupancy_v<1>(T, C, bt, bm_words, queues_global, false);
        case 4: return occupancy_v<4>(T, C, bt, bm_words, queues_global, full_pad);
        default: return 0;
    }
}

cudaError_t launch_corridor_search(cudaStream_t s, const SearchParams& p, int blocks, int bt, bool persistent,
                                   int req_base, int vm, int bm_words) {
    switch (vm) {
        case 1:
            switch (p.log_bytes) {
                case 6: return launch_v<1, PackedLog>(s, p, blocks, bt, persistent, req_base, bm_words);
                case 8: return launch_v<1, HalfLog>(s, p, blocks, bt, persistent, req_base, bm_words);
                default: return launch_v<1, WideLog>(s, p, blocks, bt, persistent, req_base, bm_words);
            }
        case 4: return launch_v<4, WideLog>(s, p, blocks, bt, persistent, req_base, bm_words);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace gmapf_b200
