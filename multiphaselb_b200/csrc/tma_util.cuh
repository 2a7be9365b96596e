// tma_util.cuh -- mbarrier and bulk-copy helpers (inline PTX) for kernels
// that stage their inputs in shared memory with the TMA unit (fused_tma.cuh).
// No multicast form is used anywhere: every copy reads this GPU's own memory
// into its own CTA.
#pragma once

#include <cuda.h>
#include <stdint.h>

#ifndef MPLB_HD
#define MPLB_HD __host__ __device__ __forceinline__
#endif

namespace mplb {

// kernel-side error flag value: a bounded wait ran out
constexpr int MPLB_KERR_WAIT = 1;
// tries of a bounded mbarrier wait (each try may suspend the thread briefly)
constexpr uint32_t TMA_WAIT_LIMIT = 1u << 22;

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_init_fence() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// add to the bytes this phase waits for, without arriving
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.expect_tx.relaxed.cta.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
// arrive once every cp.async this thread has issued so far has landed
__device__ __forceinline__ void mbar_arrive_cp_async(uint64_t* bar) {
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// 16 bytes from global to shared memory, both 16-byte aligned
__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
// true once the phase with this parity has completed
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n"
        " mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// Bounded wait: false when the phase did not complete within `limit` tries
// (each try may suspend the thread for a short, hardware-chosen time).
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t parity, uint32_t limit) {
    for (uint32_t i = 0; i < limit; i++)
        if (mbar_try_wait(bar, parity)) return true;
    return false;
}
__device__ __forceinline__ void tma_load_4d(void* dst, const CUtensorMap* map, int c0, int c1, int c2, int c3,
                                            uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];"
        ::"r"(smem_u32(dst)), "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(smem_u32(bar))
        : "memory");
}
__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, int c0, int c1, int c2, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
        ::"r"(smem_u32(dst)), "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(smem_u32(bar))
        : "memory");
}
// bulk copy of `bytes` (a multiple of 16) from global to shared memory, both 16-byte aligned
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}

// order this thread's earlier shared-memory accesses before later async-proxy (TMA) writes
__device__ __forceinline__ void fence_proxy_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// A thread of a face tile gives up at plane step j, a wait of its block having
// run out; fparity: per stage, the parity of its next wait for wrapped parts
// (that of stage j % nstage toggled already).  It takes no part in writing the
// wrapped parts of the next plane, so it arrives for them (more: there is one):
// threads that have written theirs can still see the phase complete.  Then it
// waits for the parts of plane j, the last whose bulk copies it may have in
// flight: shared memory must not be released under them.  wait() is bounded.
template <class Arrive, class Wait>
MPLB_HD void leave_face_tile(int j, int nstage, uint32_t fparity, bool more, Arrive arrive, Wait wait) {
    const int s = j % nstage;
    if (more) arrive((j + 1) % nstage);
    wait(s, ((fparity >> s) & 1u) ^ 1u);
}

// c within one extent of [0, ext): wrapped into it
MPLB_HD int wrap_any(int c, int ext) { return c < 0 ? c + ext : (c >= ext ? c - ext : c); }

// Wrapped parts of a plane stage.  A stage holds NBOX boxes of BY rows; box b
// starts at row y0 - 1 - cy_b, and every row reaches 16 bytes past the tile's
// TX columns on either side (two doubles, four floats), so in bytes all boxes
// are alike.  A tensor copy fills the parts outside the lattice with zeros;
// this writes the periodic images there: for tiles on an x face the 16 bytes
// of every row (one thread each), for tiles on a y face the one or two rows of
// a box that lie outside (one thread and one bulk copy each).  The work goes to
// the block's last warps; its first ones have the ring.  row(b, iy, y, dst,
// src, es) gives row iy of box b in shared memory, the start of lattice row y of
// its plane, and the element size; cy(b) is the box's shift; copy(dst, src)
// copies 16 bytes, bulk(dst, src, bytes) a multiple of 16.
template <int TX, int TY, int NBOX, class Cy, class Row, class Copy, class Bulk>
MPLB_HD void patch_wrapped(int tid, int nt, int x0, int y0, int nx, int ny, Cy cy, Row row, Copy copy, Bulk bulk) {
    constexpr int BY = TY + 2, NROWS = NBOX * BY;
    const bool left = x0 == 0, right = x0 + TX == nx;
    unsigned char* dst;
    const unsigned char* src;
    int es;
    const int t = nt - 1 - tid;
    if (left || right) {
        for (int r = t; r < NROWS; r += nt) {
            const int b = r / BY, iy = r - b * BY, y = y0 - 1 - cy(b) + iy;
            if (y < 0 || y >= ny) continue;  // a row of the second part
            row(b, iy, y, dst, src, es);
            if (left) copy(dst, src + nx * es - 16);
            if (right) copy(dst + 16 + TX * es, src);
        }
    }
    // rows outside: per box and side, at most two; the warp below the x part's
    const int yt = t - (NROWS + 31 < nt ? (NROWS + 31) / 32 * 32 : nt - 32);
    static_assert(2 * NBOX <= 32, "one lane per row");
    if (yt < 0 || yt >= 2 * NBOX) return;
    for (int side = 0; side < 2; side++) {
        if (side ? y0 + TY != ny : y0 != 0) continue;
        const int b = yt >> 1, w = yt & 1;
        if (w >= (side ? 1 - cy(b) : 1 + cy(b))) continue;
        const int iy = side ? BY - 1 - w : w;
        row(b, iy, wrap_any(y0 - 1 - cy(b) + iy, ny), dst, src, es);
        const int lo = left ? 16 : 0, hi = 32 + TX * es - (right ? 16 : 0);  // the part inside the box in x
        bulk(dst + lo, src + (x0 * es - 16 + lo), hi - lo);
        if (left) copy(dst, src + nx * es - 16);
        if (right) copy(dst + 16 + TX * es, src);
    }
}

}  // namespace mplb
