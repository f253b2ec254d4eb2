// records.cuh -- search records and edge rows (device code only).
//
// A record (`Rec`, internal.h) is one 32-byte L2 sector.  Reading or writing
// it with a single 256-bit access costs one L1 pass instead of two, and a
// whole-sector store lets L2 evict the sector without first filling the
// other half from DRAM.  Records are 32-byte aligned: every record array
// starts at an allocation (or array) boundary and holds whole records.
#pragma once

#include "internal.h"

namespace gmapf_b200 {

// the whole record, through L2 (records are written by other threads of the warp)
__device__ __forceinline__ void ld_rec(const Rec* r, int4& a, int4& b) {
    asm volatile("ld.global.cg.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(a.x), "=r"(a.y), "=r"(a.z), "=r"(a.w), "=r"(b.x), "=r"(b.y), "=r"(b.z), "=r"(b.w)
                 : "l"(r));
}

// {stamp or jump ancestor, G<<1|dir, ancestors 1..6}
__device__ __forceinline__ void st_rec(Rec* r, unsigned stamp, int gd, int a0, int a1, int a2, int a3, int a4,
                                       int a5) {
    asm volatile("st.global.cg.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(r), "r"((int)stamp), "r"(gd),
                 "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(a4), "r"(a5)
                 : "memory");
}

// Lanes without a row (index < 0) issue no access: one shared dummy row would
// make every warp of the GPU read the same sector in every round.
__device__ __forceinline__ void ld_edge_half(const EdgeHalf* rows, long long k, EdgeHalf& o) {
    asm volatile(
        "{ .reg .pred p; setp.ge.s64 p, %5, 0; mov.b32 %0, -1; mov.b32 %1, 0; mov.f32 %2, 0f00000000; mov.f32 %3, 0f00000000;"
        " @p ld.global.nc.v4.b32 {%0,%1,%2,%3}, [%4]; }"
        : "=&r"(o.e), "=&r"(o.info), "=&f"(o.x), "=&f"(o.y)
        : "l"(rows + k), "l"(k));
}

__device__ __forceinline__ void ld_edge_row(const EdgeRow* rows, int k, EdgeHalf& x, EdgeHalf& y) {
    ld_edge_half(&rows->x, k < 0 ? -1 : 2 * (long long)k, x);
    ld_edge_half(&rows->x, k < 0 ? -1 : 2 * (long long)k + 1, y);
}

// a word through L2, 0 (and no access) without `on`
__device__ __forceinline__ unsigned ld_word_if(const unsigned* p, bool on) {
    unsigned w;
    asm volatile("{ .reg .pred q; setp.ne.s32 q, %2, 0; mov.b32 %0, 0; @q ld.global.cg.b32 %0, [%1]; }"
                 : "=&r"(w)
                 : "l"(p), "r"((int)on)
                 : "memory");
    return w;
}

// the row into shared memory, asynchronously (k < 0: zeros, and nothing is read);
// copies_done waits for this thread's copies
__device__ __forceinline__ void copy_edge_row(EdgeHalf* to, const EdgeRow* rows, int k) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(to);
    const EdgeRow* from = rows + max(k, 0);
    const int bytes = k < 0 ? 0 : 16;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(&from->x), "r"(bytes) : "memory");
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d + 16), "l"(&from->y), "r"(bytes) : "memory");
}
__device__ __forceinline__ void copies_done() { asm volatile("cp.async.wait_all;" ::: "memory"); }

}  // namespace gmapf_b200
