// search_common.cuh -- what the two search kernels (search.cu, corridor.cu)
// share: the queue key, the queues' layout, the visited bitmap.
#pragma once

#include "internal.h"

namespace gmapf_b200 {
namespace {

// (F, G, id) lexicographic; gd = G << 1 | dir
__device__ __forceinline__ bool key_less(float fa, int ga, int ia, float fb, int gb, int ib) {
    // G<<1|dir with the side bit set orders and ties exactly as G does
    const int Ga = ga | 1, Gb = gb | 1;
    return fa != fb ? fa < fb : (Ga != Gb ? Ga < Gb : ia < ib);
}

// A queued node: its key (F, G<<1|dir, id).
constexpr int kEntryWords = 3;

// Per-lane sorted ring in shared memory: entry k of lane q is (F, G<<1|dir)
// as one 8-byte word at fg[k*T + q] and the node id at id[k*T + q].
struct Ring {
    int* base;
    int T;
    int q;
    int C;
    __device__ __forceinline__ int at(int k) const {  // k in [0, 2C)
        return (k >= C ? k - C : k) * T + q;
    }
    __device__ __forceinline__ int2* fg() const { return reinterpret_cast<int2*>(base); }
    __device__ __forceinline__ int* id() const { return base + 2 * C * T; }
};

// 2-bit visited state: bit 0 = claimed, bit 1 = reached from the start
__device__ __forceinline__ int bm_bits(unsigned w, int n) { return (int)((w >> ((n & 15) << 1)) & 3u); }
__device__ __forceinline__ int bm_get(const unsigned* bm, int n) { return bm_bits(bm[n >> 4], n); }

// SHARED: the bitmap is in shared memory; otherwise in global memory, set by
// a reduction that returns nothing (no register or scoreboard held for it)
template <bool SHARED>
__device__ __forceinline__ void bm_set(unsigned* bm, int n, int dir) {
    const unsigned bit = (1u | ((unsigned)dir << 1)) << ((n & 15) << 1);
    if constexpr (SHARED)
        atomicOr(bm + (n >> 4), bit);
    else
        asm volatile("red.relaxed.gpu.global.or.b32 [%0], %1;" ::"l"(bm + (n >> 4)), "r"(bit) : "memory");
}

constexpr unsigned kFull = 0xffffffffu;

__device__ __forceinline__ unsigned long long global_timer_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Serving ring: publish query q's completion after its results (lane 0,
// after the warp's writes are ordered by __syncwarp)
__device__ __forceinline__ void ring_complete(const SearchParams& p, int slot_row, int q, int found) {
    __threadfence_system();
    reinterpret_cast<volatile unsigned long long*>(p.done)[slot_row] =
        ((unsigned long long)(unsigned)(q + 1) << 1) | (unsigned long long)(found ? 1 : 0);
}

// per-warp shared-memory regions in 4-byte words, rounded to 16 bytes
__host__ __device__ __forceinline__ size_t search_queue_words(int C, int T) {
    return ((size_t)kEntryWords * C * T + 3) & ~(size_t)3;
}
// Path output: depth d of the start side at out[d - 1] (d >= 1), depth d of
// the target side at out[gS + gT - d] (d >= 0).
__device__ __forceinline__ int path_pos(int side, int d, int gS, int gT) {
    return side == 0 ? d - 1 : gS + gT - d;
}

}  // namespace
}  // namespace gmapf_b200
