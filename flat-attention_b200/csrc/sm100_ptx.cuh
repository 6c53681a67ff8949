// Thin inline-PTX wrappers for the Blackwell (sm_100a) primitives the tensor-core kernels use:
// mbarriers with bounded waits, TMA tiled loads, TMEM allocation, tcgen05.mma / ld / st / commit,
// and the shared-memory matrix / instruction descriptors.  No multicast qualifier is used anywhere.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>

#include <cstdint>

namespace flat {
namespace sm100 {

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// ---- warp roles ------------------------------------------------------------------------------
// The warp's index as a value the compiler knows to be the same in all lanes.
__device__ __forceinline__ int warp_index_uniform() { return __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0); }
// One lane of a converged warp.  The branch that issues tcgen05 / TMA instructions is taken on this and not on
// `lane == 0`: the compiler then knows that a single thread is active and keeps descriptors, TMEM and barrier addresses
// in uniform registers, which those instructions read; behind `lane == 0` every operand is moved over for every
// instruction (back-to-back MMAs of 128 x 64 x 16 issue every 31 clk instead of every 45, and the forward kernel of a
// B=4, 32/8 heads, N=4096, D=128 causal call takes 505 us instead of 540).
__device__ __forceinline__ bool elect_one() {
    uint32_t r;
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "elect.sync _|p, 0xffffffff;\n"
        "selp.u32 %0, 1, 0, p;\n"
        "}\n"
        : "=r"(r));
    return r != 0;
}

// ---- mbarrier --------------------------------------------------------------------------------
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_fence_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n"
        "}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
// The same test, but the thread may stay suspended in hardware for up to `hint_ns` nanoseconds while the phase
// is incomplete: a waiting warp then leaves the issue slots to the warps that compute.
__device__ __forceinline__ bool mbar_try_wait_suspend(uint32_t bar, uint32_t parity, uint32_t hint_ns) {
    uint32_t ok;
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n"
        "selp.u32 %0, 1, 0, p;\n"
        "}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity), "r"(hint_ns)
        : "memory");
    return ok != 0;
}

// Bounded wait: gives up after `kWaitCycles` clock cycles (about a second), or as soon as another thread of the CTA
// has given up (`*abort_flag != 0`).  Returns false on give-up; the caller records where and
// leaves its loop, so the kernel always terminates and the context stays usable.
constexpr uint32_t kWaitCycles = 2000000000u;  // about one second (32-bit cycle counter, wrap-safe difference)
constexpr uint32_t kSuspendNs = 20000;         // one suspended poll lasts at most 20 us
__device__ __forceinline__ bool mbar_wait_slow(uint32_t bar, uint32_t parity, volatile int *abort_flag) {
    const uint32_t start = (uint32_t)clock();
    do {
        if (mbar_try_wait_suspend(bar, parity, kSuspendNs)) return true;
    } while (*abort_flag == 0 && (uint32_t)clock() - start <= kWaitCycles);
    *abort_flag = 1;
    return false;
}
// For a thread on its own.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int *abort_flag) {
    return mbar_try_wait(bar, parity) || mbar_wait_slow(bar, parity, abort_flag);
}
// For a whole warp, all of whose lanes get the same answer: one lane may see the phase, or the abort flag, when another does
// not, and a warp of which a part leaves its loop hangs at the next instruction that takes all of it (tcgen05.ld, __syncwarp).
__device__ __forceinline__ bool mbar_wait_warp(uint32_t bar, uint32_t parity, volatile int *abort_flag) {
    return __all_sync(0xffffffffu, mbar_try_wait(bar, parity)) || __all_sync(0xffffffffu, mbar_wait_slow(bar, parity, abort_flag));
}
// For two phases at once, with one reduction.
__device__ __forceinline__ bool mbar_wait_warp(uint32_t bar0, uint32_t parity0, uint32_t bar1, uint32_t parity1, volatile int *abort_flag) {
    return __all_sync(0xffffffffu, mbar_try_wait(bar0, parity0) && mbar_try_wait(bar1, parity1)) ||
           __all_sync(0xffffffffu, mbar_wait_slow(bar0, parity0, abort_flag) && mbar_wait_slow(bar1, parity1, abort_flag));
}

// ---- TMA -------------------------------------------------------------------------------------
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

__device__ __forceinline__ void tma_load_4d(uint32_t dst, const CUtensorMap *map, int c0, int c1, int c2, int c3,
                                            uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];"
        ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(bar)
        : "memory");
}
// Tiled bulk store of one box from shared memory to global memory (bulk async-group completion).
__device__ __forceinline__ void tma_store_4d(const CUtensorMap *map, int c0, int c1, int c2, int c3, uint32_t src) {
    asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.tile.bulk_group [%0, {%1, %2, %3, %4}], [%5];" ::"l"(
                     reinterpret_cast<uint64_t>(map)),
                 "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(src)
                 : "memory");
}
__device__ __forceinline__ void bulk_commit_group() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
// the committed groups have finished READING their shared-memory sources
__device__ __forceinline__ void bulk_wait_group_read0() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }

__device__ __forceinline__ void tma_prefetch_desc(const CUtensorMap *map) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(map)) : "memory");
}

// ---- TMEM ------------------------------------------------------------------------------------
__device__ __forceinline__ void tmem_alloc(uint32_t smem_dst, uint32_t cols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_dst), "r"(cols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t cols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tc_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// The mbarrier receives one arrival when every tcgen05 operation this thread issued before has completed.
__device__ __forceinline__ void tc_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

// D[tmem] (+)= A[smem] * B[smem] and A[tmem] * B[smem].  A descriptor is base + offset, formed inside the asm block (offset in
// 16-byte units, added to the start-address field): an unrolled issue sequence then keeps only the base descriptors in
// registers.
__device__ __forceinline__ void mma_ss_off(uint32_t d_tmem, uint64_t a_base, uint64_t b_base, uint32_t off16, uint32_t idesc,
                                           uint32_t accumulate) {
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        ".reg .b64 da, db, o;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "cvt.u64.u32 o, %5;\n"
        "add.s64 da, %1, o;\n"
        "add.s64 db, %2, o;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %3, p;\n"
        "}\n" ::"r"(d_tmem), "l"(a_base), "l"(b_base), "r"(idesc), "r"(accumulate), "r"(off16)
        : "memory");
}
__device__ __forceinline__ void mma_ts_off(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_base, uint32_t off16, uint32_t idesc,
                                           uint32_t accumulate) {
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        ".reg .b64 db, o;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "cvt.u64.u32 o, %5;\n"
        "add.s64 db, %2, o;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %3, p;\n"
        "}\n" ::"r"(d_tmem), "r"(a_tmem), "l"(b_base), "r"(idesc), "r"(accumulate), "r"(off16)
        : "memory");
}

// The same with the descriptors given by their low words (start address and leading byte offset; `kDescHi1024` is the high word
// of a 128-byte-swizzled operand whose stride byte offset is 1024): half the registers and additions per instruction.
constexpr uint32_t kDescHi1024 = (1024u >> 4) | (1u << 14) | (2u << 29);
__device__ __forceinline__ void mma_ss_lo(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t off16, uint32_t idesc,
                                          uint32_t accumulate) {
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        ".reg .b32 la, lb;\n"
        ".reg .b64 da, db;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "add.u32 la, %1, %5;\n"
        "add.u32 lb, %2, %5;\n"
        "mov.b64 da, {la, %6};\n"
        "mov.b64 db, {lb, %6};\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %3, p;\n"
        "}\n" ::"r"(d_tmem), "r"(a_lo), "r"(b_lo), "r"(idesc), "r"(accumulate), "r"(off16), "n"(kDescHi1024)
        : "memory");
}
__device__ __forceinline__ void mma_ts_lo(uint32_t d_tmem, uint32_t a_tmem, uint32_t b_lo, uint32_t off16, uint32_t idesc,
                                          uint32_t accumulate) {
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        ".reg .b32 lb;\n"
        ".reg .b64 db;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "add.u32 lb, %2, %5;\n"
        "mov.b64 db, {lb, %6};\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %3, p;\n"
        "}\n" ::"r"(d_tmem), "r"(a_tmem), "r"(b_lo), "r"(idesc), "r"(accumulate), "r"(off16), "n"(kDescHi1024)
        : "memory");
}

// 32 lanes x 32 consecutive 32-bit columns: thread t of the warp reads lane (lane_base + t).
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t *r) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
          "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t *r) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t *r) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
        "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(taddr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
        "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]),
        "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]),
        "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
        : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t *r) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(taddr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
        "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}

// ---- descriptors -----------------------------------------------------------------------------
// Shared-memory matrix descriptor, 128-byte swizzle (the layout TMA writes with SWIZZLE_128B):
// bits 0-13 start address >> 4, 16-29 leading byte offset >> 4, 32-45 stride byte offset >> 4,
// 46-47 descriptor version (1 on sm_100), 61-63 layout type (2 = 128-byte swizzle).
//  K-major operand (rows of 64 16-bit elements = 128 B): SBO = 1024 (8 rows), LBO unused.
//  MN-major operand (64 contiguous elements along M/N per 128-B row, rows step along K):
//    SBO = 1024 (8 K-rows), LBO = distance between consecutive 64-element M/N blocks.
__device__ __forceinline__ uint64_t make_smem_desc(uint32_t smem_addr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
    uint64_t d = 0;
    d |= static_cast<uint64_t>((smem_addr & 0x3FFFFu) >> 4);
    d |= static_cast<uint64_t>((lbo_bytes >> 4) & 0x3FFFu) << 16;
    d |= static_cast<uint64_t>((sbo_bytes >> 4) & 0x3FFFu) << 32;
    d |= static_cast<uint64_t>(1) << 46;
    d |= static_cast<uint64_t>(2) << 61;
    return d;
}

// Instruction descriptor for kind::f16: bits 4-5 accumulator format (1 = f32), 7-9 A format,
// 10-12 B format (0 = f16, 1 = bf16), 15 A major, 16 B major (0 = K-major, 1 = MN-major),
// 17-22 N >> 3, 24-28 M >> 4.
constexpr uint32_t kFmtF16 = 0, kFmtBF16 = 1;
__host__ __device__ constexpr uint32_t make_idesc(uint32_t a_fmt, uint32_t b_fmt, uint32_t a_mn_major,
                                                  uint32_t b_mn_major, uint32_t m, uint32_t n) {
    return (1u << 4) | (a_fmt << 7) | (b_fmt << 10) | (a_mn_major << 15) | (b_mn_major << 16) | ((n >> 3) << 17) |
           ((m >> 4) << 24);
}

__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

}  // namespace sm100
}  // namespace flat
