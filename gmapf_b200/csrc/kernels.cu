// kernels.cu -- request compaction, target upload and the agents mover.
//
// Reference kernels restated here:
//   KernelFindRequests        include/gmapf/PathFinder.h:76-117
//   KernelFindMovingAgents    include/gmapf/AgentsMover.h:29-49
//   KernelMoveAgents          include/gmapf/AgentsMover.h:51-71
//   KernelResolveCollisions   include/gmapf/AgentsMover.h:73-129
//   KernelUpdatePathProgress  include/gmapf/AgentsMover.h:131-177
// Agents are stored as structure-of-arrays.  Compaction is stable (requests
// in ascending agent id).  Collisions read one snapshot of the positions
// after the move and write a second buffer (Jacobi); each agent sums its
// contributions in ascending neighbour id, found through a uniform grid whose
// cells are at least 1.0625 collision distances wide, so
// the 3x3 neighbourhood holds every agent the reference's all-pairs loop
// would accept.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "internal.h"

namespace gmapf_b200 {

namespace {

namespace cg = cooperative_groups;

constexpr int kOrderBuckets = 1024;  // of the longest-first order
constexpr int kCompactThreads = 1024;
constexpr int kBesideThreads = 256;  // beside served searches
constexpr int kCompactRun = 4;       // consecutive agents per thread and step
constexpr int kCompactCluster = 8;   // thread blocks (one cluster) for more agents than one block's step

// inclusive block scan (TH threads) of v; *total gets the sum.  warp_tot: 32 words
template <int TH>
__device__ __forceinline__ int block_scan(int v, int* warp_tot, int* total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += t;
    }
    __syncthreads();  // the previous scan's totals are read
    if (lane == 31) warp_tot[warp] = v;
    __syncthreads();
    int w = TH == 1024 || lane < TH / 32 ? warp_tot[lane] : 0;
    for (int o = 1; o < 32; o <<= 1) {  // (every warp scans the totals: no second barrier)
        const int t = __shfl_up_sync(0xffffffffu, w, o);
        if (lane >= o) w += t;
    }
    *total = __shfl_sync(0xffffffffu, w, 31);
    const int before = __shfl_sync(0xffffffffu, w, warp > 0 ? warp - 1 : 0);
    return v + (warp > 0 ? before : 0);
}

// block_scan over the cluster's blocks (CL of them) in rank order; cluster_tot:
// CL words of shared memory, read by the other blocks
template <int CL, int TH>
__device__ __forceinline__ int cluster_scan(int v, int* warp_tot, int* cluster_tot, int* total) {
    int tot;
    const int incl = block_scan<TH>(v, warp_tot, &tot);
    if constexpr (CL == 1) {
        *total = tot;
        return incl;
    } else {
        cg::cluster_group cl = cg::this_cluster();
        cl.sync();  // the previous scan's totals are read
        if (threadIdx.x < CL) cl.map_shared_rank(cluster_tot, threadIdx.x)[cl.block_rank()] = tot;
        cl.sync();
        int before = 0, all = 0;
#pragma unroll
        for (int k = 0; k < CL; k++) {
            const int t = cluster_tot[k];
            before += k < (int)cl.block_rank() ? t : 0;
            all += t;
        }
        *total = all;
        return before + incl;
    }
}

// Request compaction: four agents per thread and step, one scan of both counts
// (Search agents in the low half, Move agents in the high half: at most 32,768
// of each per step).  It reads and writes 10 to 40 bytes per agent and is bound
// by latency: loads, scan, stores, one after the other.  One block of 4,096
// agents a step up to that many, beyond it a cluster of eight blocks whose
// totals go through distributed shared memory, 32,768 agents a step: 7.9 us for
// 16,384 requests and 10.4 us for 24,000 agents in 64 scenes.  (One block with
// one agent per thread and three barriers per scan took 29 and 63 us; the same
// block with 16 agents per thread 34 and 23 us.)
//
// While a context serves, the blocks have 256 threads (1,024 agents a step in one
// block, 8,192 in the cluster): a frame starts while searches fill the SMs, and
// what serving leaves of an SM, one search block's share (24,576 registers beside
// blocks of 256, 14,336 beside blocks of 128), has room for 256 threads of 49
// registers, not for 1,024.  The frame after a burst of 8,192 retargets on the 64x64
// maze at T=8 took 4.4 ms with blocks of 1,024 threads, 0.14 now.
//
// Per-scene request limits (a scene batch): scene s takes its Search agents in
// ascending id up to P[s] (each scene is its own PathFinder, PathFinder.h:76-117).
// first[s] records how many Search agents precede the scene's first agent.
template <int CL, int TH>
__device__ __forceinline__ void compact(int A, int* state, const int* cur, const int* targ, int P, const CompactScenes& scn,
                                        int4* req, int* req_count, unsigned char* in_move, int* mv_count, int* parity,
                                        int* work_ctr, int* hist, unsigned long long* stats, const FrameWords& words) {
    __shared__ int warp_tot[32];
    __shared__ int cluster_tot[CL];
    const int tid = threadIdx.x;
    const int rank = CL > 1 ? (int)blockIdx.x : 0;
    const bool scenes = scn.agent_scene != nullptr;
    if (hist && rank == 0)  // the order's buckets
        for (int k = tid; k < kOrderBuckets; k += TH) hist[k] = 0;
    const float dt = tid == 0 && rank == 0 ? *reinterpret_cast<const volatile float*>(words.dt_host) : 0.f;
    int base_s = 0, base_m = 0, base_o = 0;  // before this step (the same on every thread)
    for (int b = 0; b < A; b += CL * TH * kCompactRun) {
        const int i0 = b + (rank * TH + tid) * kCompactRun;
        const int cnt = max(0, min(kCompactRun, A - i0));
        int st[kCompactRun], cu[kCompactRun], ta[kCompactRun];
        if (cnt == kCompactRun) {  // (runs of 4 start on 16-byte boundaries)
            auto load = [&](const int* from, int* to) {
                const int4 q = *reinterpret_cast<const int4*>(from + i0);
                to[0] = q.x;
                to[1] = q.y;
                to[2] = q.z;
                to[3] = q.w;
            };
            load(state, st);
            load(cur, cu);
            load(targ, ta);
        } else {
#pragma unroll
            for (int j = 0; j < kCompactRun; j++) {
                st[j] = j < cnt ? state[i0 + j] : GMAPF_AGENT_IDLE;
                cu[j] = j < cnt ? cur[i0 + j] : 0;
                ta[j] = j < cnt ? targ[i0 + j] : 0;
            }
        }
        bool want[kCompactRun];
        int ns = 0, nm = 0;
        unsigned flags = 0;
#pragma unroll
        for (int j = 0; j < kCompactRun; j++) {
            want[j] = st[j] == GMAPF_AGENT_SEARCH && cu[j] != ta[j];
            if (st[j] == GMAPF_AGENT_SEARCH && !want[j]) state[i0 + j] = GMAPF_AGENT_IDLE;  // PathFinder.h:91-95
            const bool m = st[j] == GMAPF_AGENT_MOVE;
            ns += want[j];
            nm += m;
            flags |= (m ? 1u : 0u) << (8 * j);
        }
        if (cnt == kCompactRun)
            *reinterpret_cast<unsigned*>(in_move + i0) = flags;
        else
            for (int j = 0; j < cnt; j++) in_move[i0 + j] = (flags >> (8 * j)) & 1u;
        int tot;
        const int incl = cluster_scan<CL, TH>(ns | nm << 16, warp_tot, cluster_tot, &tot);
        int pos = base_s + (incl & 0xffff) - ns;  // Search agents before this run
        if (!scenes) {
#pragma unroll
            for (int j = 0; j < kCompactRun; j++)
                if (want[j]) {
                    if (pos < P) req[pos] = make_int4(i0 + j, cu[j], ta[j], i0 + j);  // over capacity: stays Search
                    pos++;
                }
        } else {
            int sidx[kCompactRun], at[kCompactRun];
#pragma unroll
            for (int j = 0; j < kCompactRun; j++) {
                sidx[j] = j < cnt ? scn.agent_scene[i0 + j] : 0;
                at[j] = pos;
                if (j < cnt && i0 + j == scn.abase[sidx[j]]) scn.first[sidx[j]] = pos;
                pos += want[j];
            }
            if constexpr (CL == 1)
                __syncthreads();
            else
                cg::this_cluster().sync();
            int ok = 0;
#pragma unroll
            for (int j = 0; j < kCompactRun; j++) {
                want[j] = want[j] && at[j] - __ldcg(scn.first + sidx[j]) < scn.P[sidx[j]];
                ok += want[j];
            }
            int tot_o;
            int opos = base_o + cluster_scan<CL, TH>(ok, warp_tot, cluster_tot, &tot_o) - ok;
#pragma unroll
            for (int j = 0; j < kCompactRun; j++)
                if (want[j]) req[opos++] = make_int4(i0 + j, cu[j], ta[j], i0 + j);
            base_o += tot_o;
        }
        base_s += tot & 0xffff;
        base_m += (int)((unsigned)tot >> 16);
    }
    if (tid == 0 && rank == 0) {
        const int R = scenes ? base_o : (base_s < P ? base_s : P);
        *req_count = R;
        *mv_count = base_m;
        if (parity[1]) {  // the mover has used its grid since: the other copy's turn
            parity[0] ^= 1;
            parity[1] = 0;
        }
        *work_ctr = 0;
        *words.dt = dt;
        *words.err = 0;
        stats[ST_REQUESTS] += (unsigned long long)R;
        stats[ST_MOVING] += (unsigned long long)base_m;
    }
    if constexpr (CL > 1) cg::this_cluster().sync();  // no block leaves while another may still write its totals
}

#define COMPACT_ARGS                                                                                          \
    int A, int *state, const int *cur, const int *targ, int P, CompactScenes scn, int4 *req, int *req_count, \
        unsigned char *in_move, int *mv_count, int *parity, int *work_ctr, int *hist, unsigned long long *stats, FrameWords words
template <int TH>
__global__ void __launch_bounds__(TH) k_compact(COMPACT_ARGS) {
    compact<1, TH>(A, state, cur, targ, P, scn, req, req_count, in_move, mv_count, parity, work_ctr, hist, stats, words);
}
template <int TH>
__global__ void __cluster_dims__(kCompactCluster, 1, 1) __launch_bounds__(TH, TH == kBesideThreads ? 5 : 1)
    k_compact_cluster(COMPACT_ARGS) {
    compact<kCompactCluster, TH>(A, state, cur, targ, P, scn, req, req_count, in_move, mv_count, parity, work_ctr, hist, stats, words);
}
#undef COMPACT_ARGS

__global__ void k_apply_targets(const int4* recs, int n, int* state, int* targ_node,
                                float2* targ_pos) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const int4 r = recs[k];  // {agent, node, x bits, y bits}
    state[r.x] = GMAPF_AGENT_SEARCH;
    targ_node[r.x] = r.y;
    targ_pos[r.x] = make_float2(__int_as_float(r.z), __int_as_float(r.w));
}

// device-resident retargets: locate each target on the device (the host
// path's CuNodesMap::TryGetNodeIdx rule) and mark the agent Search
__global__ void k_apply_targets_device(const int* ids, const float2* pos, int n, int id_base, int id_count,
                                       const ScenePar* sc, const int* agent_scene, int* state, int* targ_node,
                                       float2* targ_pos, int* err) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const int lid = ids[k];
    const float2 p = pos[k];
    if (lid < 0 || lid >= id_count) {
        atomicOr(err, ERR_BAD_REQUEST);
        return;
    }
    const int id = id_base + lid;
    const int node = locate(sc[agent_scene ? agent_scene[id] : 0].loc, p.x, p.y);
    if (node < 0) {
        atomicOr(err, ERR_BAD_REQUEST);
        return;
    }
    state[id] = GMAPF_AGENT_SEARCH;
    targ_node[id] = node;
    targ_pos[id] = p;
}

__global__ void k_prepare_batch(const int* starts, const int* targets, int n, int nodes, int4* req,
                                int* req_count, int* work_ctr, int* hist, int* err) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (hist && blockIdx.x == 0)  // the order's buckets
        for (int j = threadIdx.x; j < kOrderBuckets; j += blockDim.x) hist[j] = 0;
    if (k == 0) {
        *req_count = n;
        *work_ctr = 0;
    }
    if (k >= n) return;
    int s = starts[k], t = targets[k];
    if (s < 0 || s >= nodes || t < 0 || t >= nodes) atomicOr(err, ERR_BAD_REQUEST);
    req[k] = make_int4(-1, s, t, k);
}

// Orders requests longest-first for the persistent search: the estimate is
// the landmark lower bound on the hop distance, max_l |d_l(s) - d_l(t)|, and
// requests are bucketed by it in descending order.  Results do not depend
// on the order (every request writes only its own row and agent).
//
// Two launches over all SMs (16 scattered 2-byte reads per request, then one
// read and one write of it): one block for all requests took 80 us at 16,384
// requests and 11.5 us at 2,048, now 8.6 + 4.7 and 2.7.  The buckets are scaled by the
// map's largest landmark distance, so that no pass over the estimates has to
// find their maximum first.  With a search slot for every request the order is
// of no use: they are copied.
__global__ void __launch_bounds__(128) k_order_keys(const int4* req_in, const int* req_count, int4* req_out, int2* keys,
                                                    int* hist, const unsigned short* lm, int L, int n, int lm_max,
                                                    int slots) {
    const int R = *req_count;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < R; i += gridDim.x * blockDim.x) {
        const int4 q = req_in[i];
        if (R <= slots) {
            req_out[i] = q;
            continue;
        }
        int est = 0;
        if (q.y >= 0 && q.y < n && q.z >= 0 && q.z < n) {
#pragma unroll 8
            for (int l = 0; l < L; l++) {
                const int a = lm[(size_t)l * n + q.y], b = lm[(size_t)l * n + q.z];
                const int e = (a == 65535 || b == 65535) ? 65535 : abs(a - b);
                est = max(est, e);
            }
        }
        const int b = (kOrderBuckets - 1) - (int)((long long)min(est, lm_max) * (kOrderBuckets - 1) / lm_max);
        keys[i] = make_int2(b, atomicAdd(hist + b, 1));
    }
}

__global__ void __launch_bounds__(256) k_order_place(const int4* req_in, const int* req_count, int4* req_out,
                                                     const int2* keys, const int* hist, int slots) {
    __shared__ int warp_tot[32];
    __shared__ int4 start4[kOrderBuckets / 4];
    static_assert(kOrderBuckets == 4 * 256, "four buckets per thread");
    const int* start = reinterpret_cast<const int*>(start4);
    const int R = *req_count;
    if (R <= slots) return;
    const int4 h = reinterpret_cast<const int4*>(hist)[threadIdx.x];
    const int four = h.x + h.y + h.z + h.w;
    int tot;
    const int before = block_scan<256>(four, warp_tot, &tot) - four;
    start4[threadIdx.x] = make_int4(before, before + h.x, before + h.x + h.y, before + h.x + h.y + h.z);
    __syncthreads();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < R; i += gridDim.x * blockDim.x) {
        const int2 k = keys[i];
        req_out[start[k.x] + k.y] = req_in[i];
    }
}

// The agent grid of a frame: per cell a count and, for the agents beyond the
// four of its bucket, four lists that they join in turn.  Cells hold about
// one agent on average (5% of the agents of a uniform crowd find their bucket
// full), so one 16-byte read gives a cell's agents, and binning is one pass: no
// scan over the cells and no second pass to place the agents (k_cell_scan and
// k_scatter took 4 + 4 us at 2,048 agents, 39 + 4 us at 24,000 in 64 scenes).
// Two copies of the counts take turns, so that a frame's binning clears the
// other frame's without a launch of its own; *p.parity says whose turn it is (the
// compaction switches it once the collision pass has marked the copy as used).
// The buckets and the lists' heads are not cleared: the count says how many
// entries each holds.
//
// Where a crowd gathers a cell holds hundreds.  Its four lists are followed
// together, as each step of a list waits for the one before: the mover of 4,096
// agents within 118 units of one place (2,000 agents in the nine cells of each) takes
// 3.4 ms, with one list per cell 4.5, with the cells' agents sorted into runs 4.0.
constexpr int kBucket = 4, kLists = 4;

// move (AgentsMover.h:51-71) fused with the binning
__global__ void k_move_bin(MoverParams p) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (*p.mv_count == 0) return;  // AgentsMover.h:296-297
    const int turn = *p.parity & 1;
    int* const old = p.cell_count + (size_t)(1 - turn) * p.cells;
    for (int k = i; k < p.cells; k += gridDim.x * blockDim.x) old[k] = 0;
    if (i >= p.A) return;
    const ScenePar& sc = p.sc[p.agent_scene ? p.agent_scene[i] : 0];
    float2 c = p.pos[i];
    const float step = GM_FMUL(sc.speed, *p.dt);
    if (p.in_move[i] && p.step_idx[i] != -1) {
        const float2 s = p.step_pos[i];
        const float dx = GM_FSUB(s.x, c.x), dy = GM_FSUB(s.y, c.y);
        const float len = GM_FSQRT(GM_FADD(GM_FMUL(dx, dx), GM_FMUL(dy, dy)));
        if (len <= step) {
            c = s;
        } else {
            c.x = GM_FADD(c.x, GM_FMUL(GM_FDIV(dx, len), step));
            c.y = GM_FADD(c.y, GM_FMUL(GM_FDIV(dy, len), step));
        }
    }
    p.pos_mid[i] = c;
    int cell = -1;
    if (gm_isfinite(c.x) && gm_isfinite(c.y)) {
        const int cx = grid_cell(c.x, sc.ax0, sc.ainv, sc.aw);
        const int cy = grid_cell(c.y, sc.ay0, sc.ainv, sc.ah);
        cell = sc.cell_base + cy * sc.aw + cx;
        const int k = atomicAdd(p.cell_count + (size_t)turn * p.cells + cell, 1);
        if (k < kBucket)
            p.bucket[kBucket * (size_t)cell + k] = i;
        else  // (the first of a list takes what an earlier frame left as its next, which is never followed)
            p.next[i] = atomicExch(p.lists + kLists * (size_t)cell + (k & (kLists - 1)), i);
    }
    p.cell_of[i] = cell;
}

// f(agent, its position) for the first min(n, 4) of q
template <class F>
__device__ __forceinline__ void each_of(const MoverParams& p, int4 q, int n, const F& f) {
    const int j[4] = {q.x, q.y, q.z, q.w};
    float2 o[4];
#pragma unroll
    for (int m = 0; m < 4; m++) o[m] = m < n ? p.pos_mid[j[m]] : make_float2(0.f, 0.f);
#pragma unroll
    for (int m = 0; m < 4; m++)
        if (m < n) f(j[m], o[m]);
}

// the same for the `n` agents of a cell beyond its bucket: list m holds those
// numbered m, m + 4, ... of them (a step reads no further than its list goes)
template <class F>
__device__ __forceinline__ void each_beyond(const MoverParams& p, int cell, int n, const F& f) {
    int4 q = *reinterpret_cast<const int4*>(p.lists + kLists * (size_t)cell);
    for (; n > 0; n -= kLists) {
        const int4 r = make_int4(n > 4 ? p.next[q.x] : 0, n > 5 ? p.next[q.y] : 0, n > 6 ? p.next[q.z] : 0,
                                 n > 7 ? p.next[q.w] : 0);
        each_of(p, q, n, f);
        q = r;
    }
}

constexpr int kMaxLocal = 16;

// The agents pushing one agent, with their contributions, ids ascending
struct Pushes {
    int ids[kMaxLocal];
    float vx[kMaxLocal], vy[kMaxLocal];
    int cnt = 0;
    bool overflow = false;
    __device__ __forceinline__ void add(int j, float dx, float dy, float d2, float cd) {
        if (cnt >= kMaxLocal) {
            overflow = true;
            return;
        }
        const float d = GM_FSQRT(d2);
        const float shift = GM_FSUB(cd, d);
        const float x = GM_FMUL(GM_FDIV(dx, d), shift);
        const float y = GM_FMUL(GM_FDIV(dy, d), shift);
        int k = cnt++;
        while (k > 0 && ids[k - 1] > j) {
            ids[k] = ids[k - 1];
            vx[k] = vx[k - 1];
            vy[k] = vy[k - 1];
            k--;
        }
        ids[k] = j;
        vx[k] = x;
        vy[k] = y;
    }
};

// collisions (AgentsMover.h:73-129) + path progress (AgentsMover.h:131-177)
//
// One agent per thread, bound by its chain of dependent reads, not by their
// number: the nine cells' counts are read together, then their buckets, then the
// positions of a row of cells, and what the path progress needs is read at the
// start.  One cell after the other (start, end, items, positions: 27 reads in a
// row) took 22 us at 2,048 agents under ncu.  Blocks of 64 spread a small crowd over the
// SMs.
__global__ void __launch_bounds__(64, 8) k_collide_progress(MoverParams p) {
    if (*p.mv_count == 0) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= p.A) return;
    if (i == 0) p.parity[1] = 1;
    const ScenePar& sc = p.sc[p.agent_scene ? p.agent_scene[i] : 0];
    const float2 me = p.pos_mid[i];
    const int c = p.cell_of[i];
    const bool moving = p.in_move[i];
    const int L = p.path_len[i];
    int si = p.step_idx[i];
    const int sn = p.step_node[i];
    const float2 step_pos = p.step_pos[i];
    const int* const counts = p.cell_count + (size_t)(*p.parity & 1) * p.cells;
    float2 tri[3];  // the step's triangle
    if (moving && sn >= 0 && sn < p.n) {
#pragma unroll
        for (int k = 0; k < 3; k++) tri[k] = p.tri[3 * (size_t)sn + k];
    }
    float2 np = me;
    unsigned examined = 0;  // agents of the 3x3 cells read (the agent itself included)
    if (c >= 0) {
        const int lc = c - sc.cell_base;  // cell within the agent's scene
        const int cx = lc % sc.aw, cy = lc / sc.aw;
        int h[9];
        int4 b[9];
        unsigned over = 0;  // cells with agents beyond their bucket
#pragma unroll
        for (int k = 0; k < 9; k++) {
            const int x = cx + k % 3 - 1, y = cy + k / 3 - 1;
            const bool in = x >= 0 && x < sc.aw && y >= 0 && y < sc.ah;
            h[k] = in ? counts[sc.cell_base + y * sc.aw + x] : 0;
        }
#pragma unroll
        for (int k = 0; k < 9; k++) {
            examined += h[k];
            over |= (h[k] > kBucket ? 1u : 0u) << k;
            b[k] = make_int4(-1, -1, -1, -1);
            if (h[k] > 0)
                b[k] = *reinterpret_cast<const int4*>(p.bucket + kBucket * (size_t)(c + (k / 3 - 1) * sc.aw + k % 3 - 1));
            // (entries beyond the count are a former frame's)
            if (h[k] < 2) b[k].y = -1;
            if (h[k] < 3) b[k].z = -1;
            if (h[k] < 4) b[k].w = -1;
        }
        Pushes ps;
        auto meet = [&](int j, float2 o) {
            const float dx = GM_FSUB(me.x, o.x), dy = GM_FSUB(me.y, o.y);
            const float d2 = GM_FADD(GM_FMUL(dx, dx), GM_FMUL(dy, dy));
            if (d2 < sc.cd2) ps.add(j, dx, dy, d2, sc.cd);
        };
#pragma unroll
        for (int r = 0; r < 3; r++) {
            int id[12];
            float2 o[12];
#pragma unroll
            for (int k = 0; k < 3; k++) {
                id[4 * k] = b[3 * r + k].x;
                id[4 * k + 1] = b[3 * r + k].y;
                id[4 * k + 2] = b[3 * r + k].z;
                id[4 * k + 3] = b[3 * r + k].w;
            }
#pragma unroll
            for (int k = 0; k < 12; k++) {
                if (id[k] == i) id[k] = -1;
                o[k] = id[k] >= 0 ? p.pos_mid[id[k]] : make_float2(0.f, 0.f);
            }
#pragma unroll
            for (int k = 0; k < 12; k++)
                if (id[k] >= 0) meet(id[k], o[k]);
        }
        for (; over; over &= over - 1) {
            const int k = __ffs(over) - 1;
            const int cell = c + (k / 3 - 1) * sc.aw + k % 3 - 1;
            each_beyond(p, cell, counts[cell] - kBucket, [&](int j, float2 o) {
                if (j != i) meet(j, o);
            });
        }
        float sx = 0.f, sy = 0.f;
        int total = 0;
        if (!ps.overflow) {
            for (int k = 0; k < ps.cnt; k++) {
                sx = GM_FADD(sx, ps.vx[k]);
                sy = GM_FADD(sy, ps.vy[k]);
            }
            total = ps.cnt;
        } else {
            // dense crowd: take contributors in ascending id by repeated minimum search
            int last = -1;
            for (;;) {
                int best = 0x7fffffff;
                float bvx = 0.f, bvy = 0.f;
                auto look = [&](int j, float2 o) {
                    if (j == i || j <= last || j >= best) return;
                    const float dx = GM_FSUB(me.x, o.x), dy = GM_FSUB(me.y, o.y);
                    const float d2 = GM_FADD(GM_FMUL(dx, dx), GM_FMUL(dy, dy));
                    if (!(d2 < sc.cd2)) return;
                    const float d = GM_FSQRT(d2);
                    const float shift = GM_FSUB(sc.cd, d);
                    best = j;
                    bvx = GM_FMUL(GM_FDIV(dx, d), shift);
                    bvy = GM_FMUL(GM_FDIV(dy, d), shift);
                };
                for (int y = max(cy - 1, 0); y <= min(cy + 1, sc.ah - 1); y++)
                    for (int x = max(cx - 1, 0); x <= min(cx + 1, sc.aw - 1); x++) {
                        const int cc = sc.cell_base + y * sc.aw + x;
                        const int n = counts[cc];
                        if (n > 0) each_of(p, *reinterpret_cast<const int4*>(p.bucket + kBucket * (size_t)cc), n, look);
                        if (n > kBucket) each_beyond(p, cc, n - kBucket, look);
                    }
                if (best == 0x7fffffff) break;
                sx = GM_FADD(sx, bvx);
                sy = GM_FADD(sy, bvy);
                total++;
                last = best;
            }
        }
        if (total > 0) {
            const float fc = (float)total;
            const float ax = GM_FDIV(sx, fc), ay = GM_FDIV(sy, fc);
            const float rx = GM_FSUB(GM_FMUL(ax, p.cs), GM_FMUL(ay, p.sn));
            const float ry = GM_FADD(GM_FMUL(ax, p.sn), GM_FMUL(ay, p.cs));
            const float px = GM_FADD(me.x, rx), py = GM_FADD(me.y, ry);
            if (locate(sc.loc, px, py) >= 0) np = make_float2(px, py);
        }
    }
    p.pos[i] = np;
    {  // counter of the agents examined (the mover's per-agent traffic), one atomic per warp
        const unsigned m = __activemask();
        const unsigned tot = __reduce_add_sync(m, examined);
        if ((threadIdx.x & 31) == __ffs(m) - 1) atomicAdd(p.stats + ST_NEIGHBOURS, (unsigned long long)tot);
    }

    if (!moving) return;
    // path progress
    const int* path = p.paths + (long long)i * p.path_stride;
    if (si == -1) {
        if (L < 1) {
            atomicOr(p.err, ERR_BOUNDS);
            return;
        }
        const int nd = path[0];
        p.step_idx[i] = 0;
        p.step_node[i] = nd;
        p.step_pos[i] = p.waypoints ? p.waypoints[(long long)i * p.path_stride] : p.cen[nd];
        return;
    }
    if (sn < 0 || sn >= p.n) {
        atomicOr(p.err, ERR_BOUNDS);
        return;
    }
    const bool inside = point_in_tri(np.x, np.y, tri[0], tri[1], tri[2]);
    bool at_point = false;  // path smoothing: the steering point reached
    if (p.waypoints && !inside) {
        const float dx = GM_FSUB(step_pos.x, np.x), dy = GM_FSUB(step_pos.y, np.y);
        at_point = GM_FSQRT(GM_FADD(GM_FMUL(dx, dx), GM_FMUL(dy, dy))) <= sc.arrive;
    }
    if (!inside && !at_point) return;
    if (inside) {
        p.cur_node[i] = sn;
        if (si < L) si += 1;
    } else {
        // a straight run to a funnel corner may cross thin corridor triangles
        // between two frames: skip every step that steers to the same point
        const float2* wp = p.waypoints + (long long)i * p.path_stride;
        int cur = p.cur_node[i];
        while (si < L && wp[si].x == step_pos.x && wp[si].y == step_pos.y) cur = path[si++];
        p.cur_node[i] = cur;
    }
    p.step_idx[i] = si;
    if (si == L) {
        const float2 t = p.targ_pos[i];
        const float dx = GM_FSUB(t.x, np.x), dy = GM_FSUB(t.y, np.y);
        const float len = GM_FSQRT(GM_FADD(GM_FMUL(dx, dx), GM_FMUL(dy, dy)));
        if (len > sc.arrive)
            p.step_pos[i] = t;
        else
            p.state[i] = GMAPF_AGENT_IDLE;
    } else {
        const int nd = path[si];
        p.step_node[i] = nd;
        p.step_pos[i] = p.waypoints ? p.waypoints[(long long)i * p.path_stride + si] : p.cen[nd];
    }
}

// ---- path smoothing (opt-in): the simple stupid funnel (M. Mononen, 2010)
// over the corridor of a path.  Portal 0 is the agent's position, portal k
// (1..L) the edge shared by triangles k-1 and k of the corridor (triangle 0 =
// the start triangle, triangle k = path[k-1]), portal L+1 the target
// position.  Step k of the path (heading into path[k]) steers to the first
// funnel corner at a portal index >= k+1.

// twice the signed area of (a, b, c): > 0 when c lies left of a -> b
__device__ __forceinline__ float area2(float2 a, float2 b, float2 c) {
    const float bx = GM_FSUB(b.x, a.x), by = GM_FSUB(b.y, a.y);
    const float cx = GM_FSUB(c.x, a.x), cy = GM_FSUB(c.y, a.y);
    return GM_FSUB(GM_FMUL(bx, cy), GM_FMUL(cx, by));
}

__device__ __forceinline__ bool veq(float2 a, float2 b) { return a.x == b.x && a.y == b.y; }

// path smoothing 2: both ends of an edge portal moved inward by c (the agent
// radius), so that the funnel's corners keep that distance from the walls; a
// portal no wider than 2c becomes its midpoint
__device__ __forceinline__ void narrow_portal(float2& l, float2& r, float c) {
    if (!(c > 0.f)) return;
    const float dx = GM_FSUB(r.x, l.x), dy = GM_FSUB(r.y, l.y);
    const float w = GM_FSQRT(GM_FADD(GM_FMUL(dx, dx), GM_FMUL(dy, dy)));
    if (w > GM_FADD(c, c)) {
        const float t = GM_FDIV(c, w);
        const float ox = GM_FMUL(dx, t), oy = GM_FMUL(dy, t);
        l = make_float2(GM_FADD(l.x, ox), GM_FADD(l.y, oy));
        r = make_float2(GM_FSUB(r.x, ox), GM_FSUB(r.y, oy));
    } else {
        const float mx = GM_FMUL(GM_FADD(l.x, r.x), 0.5f), my = GM_FMUL(GM_FADD(l.y, r.y), 0.5f);
        l = r = make_float2(mx, my);
    }
}

// portal k as (left, right) seen travelling from triangle k-1 to triangle k;
// triangles that share no edge give their centroid as a point portal
__device__ void corridor_portal(const MoverParams& p, const int* path, int start_tri, int L, float2 sp, float2 ep,
                                int k, float clear, float2& left, float2& right) {
    if (k <= 0) {
        left = right = sp;
        return;
    }
    if (k > L) {
        left = right = ep;
        return;
    }
    const int u = k == 1 ? start_tri : path[k - 2];
    const int v = path[k - 1];
    if (u < 0 || u >= p.n || v < 0 || v >= p.n) {
        left = right = ep;
        return;
    }
    const float2* A = p.tri + 3 * (size_t)u;
    const float2* B = p.tri + 3 * (size_t)v;
    float2 s0 = make_float2(0.f, 0.f), s1 = s0;
    int cnt = 0;
    for (int a = 0; a < 3; a++) {
        const float2 va = A[a];
        if (veq(va, B[0]) || veq(va, B[1]) || veq(va, B[2])) {
            if (cnt == 0) s0 = va;
            if (cnt == 1) s1 = va;
            cnt++;
        }
    }
    if (cnt < 2) {
        left = right = p.cen[v];
        return;
    }
    if (area2(p.cen[u], p.cen[v], s0) > 0.f) {
        left = s0;
        right = s1;
    } else {
        left = s1;
        right = s0;
    }
    narrow_portal(left, right, clear);
}

// One warp per agent whose path starts this frame (in Move at the frame's
// start, step index -1): fills its path row of steering points.  The funnel is a
// serial walk along the corridor and a portal needs two rounds of dependent
// reads (the path's triangles, then their corners and centroids), so one thread
// per agent spent its time waiting for them (160 us for 2,048 agents with paths
// of 25 triangles on average).  The lanes work out 32 portals at once into
// shared memory, all lanes walk them together, and each corner's stretch of
// steering points is written by all lanes: 31 us.
constexpr int kFunnelWarps = 4;

__global__ void __launch_bounds__(32 * kFunnelWarps) k_funnel(MoverParams p) {
    __shared__ float4 window[kFunnelWarps][32];  // portals [base, base + 32): left, right
    if (*p.mv_count == 0) return;
    const int lane = threadIdx.x & 31;
    const int i = blockIdx.x * kFunnelWarps + (threadIdx.x >> 5);
    if (i >= p.A) return;
    if (!p.in_move[i] || p.step_idx[i] != -1) return;
    const int L = p.path_len[i];
    if (L < 1 || L > p.path_stride) return;
    float4* const portal = window[threadIdx.x >> 5];
    const int* path = p.paths + (long long)i * p.path_stride;
    float2* wp = p.waypoints + (long long)i * p.path_stride;
    const float2 sp = p.pos[i], ep = p.targ_pos[i];
    const int st = p.cur_node[i];
    const float clear = p.sc[p.agent_scene ? p.agent_scene[i] : 0].clear;
    float2 apex = sp, fl = sp, fr = sp;
    int apex_i = 0, left_i = 0, right_i = 0, filled = 0;
    const int max_iter = 4 * (L + 2) + 16;  // every restart moves the apex forward
    int iter = 0, base = -32;
    bool capped = false;
    auto corner = [&](float2 at, int upto) {
        for (int j = filled + lane; j < upto; j += 32) wp[j] = at;
        filled = max(filled, upto);
    };
    for (int k = 1; k <= L + 1; k++) {
        if (++iter > max_iter) {
            capped = true;
            break;
        }
        if (k < base || k >= base + 32) {
            base = k;
            __syncwarp();
            if (base + lane <= L + 1) {
                float2 l, r;
                corridor_portal(p, path, st, L, sp, ep, base + lane, clear, l, r);
                portal[lane] = make_float4(l.x, l.y, r.x, r.y);
            }
            __syncwarp();
        }
        const float4 q = portal[k - base];
        const float2 l = make_float2(q.x, q.y), r = make_float2(q.z, q.w);
        if (area2(apex, fr, r) >= 0.f) {  // right edge moves inward
            if (veq(apex, fr) || area2(apex, fl, r) < 0.f) {
                fr = r;
                right_i = k;
            } else {  // crosses the left edge: its end is a corner
                corner(fl, min(left_i, L));
                apex = fl;
                apex_i = left_i;
                fr = fl = apex;
                right_i = left_i = apex_i;
                k = apex_i;
                continue;
            }
        }
        if (area2(apex, fl, l) <= 0.f) {  // left edge moves inward
            if (veq(apex, fl) || area2(apex, fr, l) > 0.f) {
                fl = l;
                left_i = k;
            } else {  // crosses the right edge
                corner(fr, min(right_i, L));
                apex = fr;
                apex_i = right_i;
                fl = fr = apex;
                left_i = right_i = apex_i;
                k = apex_i;
                continue;
            }
        }
    }
    for (int j = filled + lane; j < L; j += 32) {
        const int nd = path[j];
        wp[j] = (capped && nd >= 0 && nd < p.n) ? p.cen[nd] : ep;
    }
}

// GMAPF.cu:227,244 -> CuNodesMap.h:53-66 for a batch of points: the first
// containing triangle in ascending id, through the point-location grid.  Blocks
// of one warp: a frame's searches leave 4,096 registers of an SM (1,024 with 28 warps
// of 72 registers), room for one or more of them and not for a block of 256, with which
// retargeting 16,384 agents during a full-retarget frame of the 160x160 maze waited
// 13 ms for searches to end (0.3 now).
constexpr int kLocateThreads = 32;
__global__ void __launch_bounds__(kLocateThreads) k_locate_points(LocateGrid g, const float2* pts, int n, int* out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = locate(g, pts[i].x, pts[i].y);
}

// one thread per directed edge (v, s); see EdgeRow
__global__ void k_edge_rows(const SearchRow* rows, int n, EdgeRow* out, EdgeHalf* third) {
    const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= 4ll * n) return;
    const int v = (int)(k >> 2), s = (int)(k & 3);
    const SearchRow r = rows[v];
    const int nb[3] = {r.n0, r.n1, r.n2};
    const float2 cen[3] = {make_float2(r.x0, r.y0), make_float2(r.x1, r.y1), make_float2(r.x2, r.y2)};
    const int parent = s < r.deg ? nb[s] : -1;
    EdgeRow o{{-1, (unsigned)r.deg << 4, 0.f, 0.f}, {-1, 0, 0.f, 0.f}};
    EdgeHalf z{-1, 0, 0.f, 0.f};
    int found = 0;
    for (int j = 0; j < r.deg; j++) {
        const int w = nb[j];
        if (w == parent) continue;
        const SearchRow& q = rows[w];
        const int back = (q.deg > 0 && q.n0 == v) ? 0 : (q.deg > 1 && q.n1 == v) ? 1 : (q.deg > 2 && q.n2 == v) ? 2 : 3;
        if (found < 2) {
            EdgeHalf& h = found == 0 ? o.x : o.y;
            h.e = w << 2 | back;
            h.info |= 1u << j;
            h.x = cen[j].x;
            h.y = cen[j].y;
        } else {
            z = EdgeHalf{w << 2 | back, 4u, cen[j].x, cen[j].y};
            o.x.info |= kEdgeThird;
        }
        found++;
    }
    out[k] = o;
    if (s == 3) third[v] = z;  // (only a row that leaves no neighbour out has a third)
}

inline int blocks_for(int n, int bt) { return (n + bt - 1) / bt; }

}  // namespace

void launch_compact(cudaStream_t s, int A, int* state, const int* cur, const int* targ, int P,
                    const CompactScenes& scn, int4* req, int* req_count, unsigned char* in_move, int* mv_count,
                    int* parity, int* work_ctr, int* hist, unsigned long long* stats, const FrameWords& words,
                    bool beside_searches) {
    const int threads = beside_searches ? kBesideThreads : kCompactThreads;
    const bool one = A <= threads * kCompactRun;
    auto kernel = beside_searches ? (one ? k_compact<kBesideThreads> : k_compact_cluster<kBesideThreads>)
                                  : (one ? k_compact<kCompactThreads> : k_compact_cluster<kCompactThreads>);
    kernel<<<one ? 1 : kCompactCluster, threads, 0, s>>>(A, state, cur, targ, P, scn, req, req_count, in_move, mv_count,
                                                         parity, work_ctr, hist, stats, words);
}

void launch_apply_targets(cudaStream_t s, const int4* recs, int n, int* state, int* targ_node,
                          float2* targ_pos) {
    if (n <= 0) return;
    k_apply_targets<<<blocks_for(n, 256), 256, 0, s>>>(recs, n, state, targ_node, targ_pos);
}

void launch_locate_points(cudaStream_t s, const LocateGrid& g, const float2* pts, int n, int* out) {
    if (n <= 0) return;
    k_locate_points<<<blocks_for(n, kLocateThreads), kLocateThreads, 0, s>>>(g, pts, n, out);
}

void launch_apply_targets_device(cudaStream_t s, const int* ids, const float2* pos, int n, int id_base,
                                 int id_count, const ScenePar* sc, const int* agent_scene, int* state,
                                 int* targ_node, float2* targ_pos, int* err) {
    if (n <= 0) return;
    k_apply_targets_device<<<blocks_for(n, 256), 256, 0, s>>>(ids, pos, n, id_base, id_count, sc, agent_scene,
                                                              state, targ_node, targ_pos, err);
}

void launch_prepare_batch(cudaStream_t s, const int* starts, const int* targets, int n, int nodes,
                          int4* req, int* req_count, int* work_ctr, int* hist, int* err) {
    k_prepare_batch<<<blocks_for(n > 0 ? n : 1, 256), 256, 0, s>>>(starts, targets, n, nodes, req,
                                                                   req_count, work_ctr, hist, err);
}

void launch_edge_rows(cudaStream_t s, const SearchRow* rows, int n, EdgeRow* out, EdgeHalf* third) {
    k_edge_rows<<<(unsigned)((4ll * n + 255) / 256), 256, 0, s>>>(rows, n, out, third);
}

void launch_order_requests(cudaStream_t s, const int4* req_in, const int* req_count, int most, int4* req_out,
                           const OrderParams& o, int n, int slots) {
    const int blocks = std::max(1, std::min(128, blocks_for(most, 256)));
    k_order_keys<<<2 * blocks, 128, 0, s>>>(req_in, req_count, req_out, o.keys, o.hist, o.lm, o.L, n, o.lm_max, slots);
    k_order_place<<<blocks, 256, 0, s>>>(req_in, req_count, req_out, o.keys, o.hist, slots);
}

void launch_move_bin(cudaStream_t s, const MoverParams& p) {
    k_move_bin<<<blocks_for(p.A, 128), 128, 0, s>>>(p);
}

void launch_funnel(cudaStream_t s, const MoverParams& p) {
    if (p.A <= 0 || !p.waypoints) return;
    k_funnel<<<blocks_for(p.A, kFunnelWarps), 32 * kFunnelWarps, 0, s>>>(p);
}

void launch_collide_progress(cudaStream_t s, const MoverParams& p) {
    k_collide_progress<<<blocks_for(p.A, 64), 64, 0, s>>>(p);
}

}  // namespace gmapf_b200
