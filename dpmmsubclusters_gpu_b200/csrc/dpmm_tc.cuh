// dpmm_tc.cuh -- tcgen05 / mbarrier / bulk-copy primitives and operand layouts shared by the tensor-core
// kernels (dpmm_tc.cu, dpmm_rows_tc.cu).
#pragma once

#include <cuda_bf16.h>

#include "dpmm_device.cuh"

namespace dpmm {
namespace tc {

constexpr int BM = 128;                    // points per tile (TMEM lanes)
constexpr int KD = 64;                     // contraction length (one 128-byte bf16 row)
constexpr int A_BYTES = BM * KD * 2;       // 16 KB (one of hi / lo)
constexpr int A_TILE = 2 * A_BYTES;        // 32 KB: hi then lo
constexpr size_t kTcSmemCap = 227 * 1024;

enum : int {
    ERR_TIMEOUT_FULL = 1, ERR_TIMEOUT_EMPTY = 2, ERR_TIMEOUT_TFULL = 3, ERR_TIMEOUT_TEMPTY = 4,
    ERR_TIMEOUT_AFULL = 5, ERR_TIMEOUT_AEMPTY = 6, ERR_TIMEOUT_BFULL = 9, ERR_TIMEOUT_BEMPTY = 10
};

__host__ __device__ constexpr uint32_t sw128_offset(int row, int k)
{
    return (uint32_t)((row >> 3) * 1024 + (row & 7) * 128 + ((((k >> 3) ^ (row & 7)) & 7) << 4) + (k & 7) * 2);
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

__device__ __forceinline__ uint64_t global_ns()
{
    uint64_t t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}

constexpr uint64_t WAIT_LIMIT_NS = 2000000000ull;   // 2 s: legitimate waits here are microseconds

// Non-blocking probe of a phase (no suspend).
__device__ __forceinline__ bool mbar_test_wait(uint64_t* bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

// Potentially blocking probe: the thread may sleep until the phase completes, for at most about
// `ns` nanoseconds (the suspend-time hint), instead of returning at once and spinning.
__device__ __forceinline__ bool mbar_try_wait_sleep(uint64_t* bar, uint32_t parity, uint32_t ns)
{
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity), "r"(ns)
        : "memory");
    return ok != 0;
}

// Single-thread bounded wait.  Gives up after WAIT_LIMIT_NS, or early when another CTA of the
// launch has already reported an error (gerr != nullptr).  Between non-blocking probes the thread
// backs off with nanosleep (32 ns growing to 256 ns), so that waiting warps do not fill the issue
// slots and the barrier / timer pipes that the working warps need.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t parity, const volatile int32_t* gerr)
{
    if (mbar_test_wait(bar, parity)) return true;
    const uint64_t t0 = global_ns();
    uint32_t sleep = 32;
    for (uint32_t i = 1;; ++i) {
        __nanosleep(sleep);
        if (mbar_test_wait(bar, parity)) return true;
        if (sleep < 256) sleep <<= 1;
        if ((i & 63) == 0) {
            if (global_ns() - t0 > WAIT_LIMIT_NS) return false;
            if (gerr && *gerr) return false;
        }
    }
}

// The same on the potentially blocking probe: the thread sleeps in hardware until the phase completes or the
// hint runs out, so a waiting role costs a few instructions instead of a poll every 32-256 ns.
__device__ __forceinline__ bool mbar_wait_blocking(uint64_t* bar, uint32_t parity, const volatile int32_t* gerr)
{
    if (mbar_try_wait_sleep(bar, parity, 2000)) return true;
    const uint64_t t0 = global_ns();
    for (uint32_t i = 1;; ++i) {
        if (mbar_try_wait_sleep(bar, parity, 2000)) return true;
        if ((i & 15) == 0) {
            if (global_ns() - t0 > WAIT_LIMIT_NS) return false;
            if (gerr && *gerr) return false;
        }
    }
}

// Warp-uniform bounded wait: lane 0 polls (one barrier operation per poll instead of 32) and
// the outcome is broadcast; __syncwarp orders the other lanes after lane 0's acquire.  All lanes
// take the same decision (the epilogue's tcgen05.ld is warp-collective).
__device__ __forceinline__ bool warp_wait_bounded(uint64_t* bar, uint32_t parity, const volatile int32_t* gerr)
{
    int ok = 1;
    if ((threadIdx.x & 31) == 0) ok = mbar_wait_bounded(bar, parity, gerr) ? 1 : 0;
    ok = __shfl_sync(0xffffffffu, ok, 0);
    __syncwarp();
    return ok != 0;
}

// The same on the blocking probe.
__device__ __forceinline__ bool warp_wait_blocking(uint64_t* bar, uint32_t parity, const volatile int32_t* gerr)
{
    int ok = 1;
    if ((threadIdx.x & 31) == 0) ok = mbar_wait_blocking(bar, parity, gerr) ? 1 : 0;
    ok = __shfl_sync(0xffffffffu, ok, 0);
    __syncwarp();
    return ok != 0;
}

// One arrival per warp: every lane's prior work is ordered before lane 0's release by __syncwarp.
__device__ __forceinline__ void warp_arrive(uint64_t* bar)
{
    __syncwarp();
    if ((threadIdx.x & 31) == 0) mbar_arrive(bar);
}

__device__ __forceinline__ void bulk_copy_g2s(void* smem_dst, const void* gmem_src, uint32_t bytes, uint64_t* bar)
{
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
            smem_u32(smem_dst)),
        "l"(gmem_src), "r"(bytes), "r"(smem_u32(bar))
        : "memory");
}

__device__ __forceinline__ uint64_t sw128_desc(uint32_t saddr)
{
    uint64_t d = 0;
    d |= (uint64_t)((saddr & 0x3FFFFu) >> 4);   // start address
    d |= (uint64_t)1 << 16;                      // leading byte offset (unused for swizzled K-major)
    d |= (uint64_t)(1024 >> 4) << 32;            // stride byte offset: 8-row atoms 1024 B apart
    d |= (uint64_t)1 << 46;                      // descriptor version (sm_100)
    d |= (uint64_t)2 << 61;                      // 128-byte swizzle
    return d;
}

// kind::f16 instruction descriptor: F32 accumulator, BF16 A and B, both K-major, M = 128, N columns
__host__ __device__ constexpr uint32_t bf16_idesc(int n)
{
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
}

__device__ __forceinline__ void umma_bf16_n(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accum)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accum)
        : "memory");
}

__device__ __forceinline__ void umma_commit(uint64_t* bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// 32 consecutive accumulator columns of this thread's TMEM lane (warp-collective)
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32])
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// Two FP32 operations in one instruction (each half rounds as the scalar one)
__device__ __forceinline__ uint64_t pack2(float lo, float hi)
{
    uint64_t d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
    return d;
}
__device__ __forceinline__ void unpack2(uint64_t v, float& lo, float& hi)
{
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c)
{
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}

__device__ __forceinline__ void bf16_split(float v, __nv_bfloat16& hi, __nv_bfloat16& lo)
{
    hi = __float2bfloat16_rn(v);
    lo = __float2bfloat16_rn(v - __bfloat162float(hi));
}

// bf16_split of four values, packed: hi and lo as 4 x BF16 (8 bytes) each
__device__ __forceinline__ uint32_t cvt_bf16x2(float lo, float hi)
{
    uint32_t d;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo));
    return d;
}

__device__ __forceinline__ void bf16_split4(float a, float b, float c, float d, uint2& hi, uint2& lo)
{
    hi = make_uint2(cvt_bf16x2(a, b), cvt_bf16x2(c, d));
    const uint64_t minus = pack2(-1.f, -1.f);   // v - hi, two at a time
    float r0, r1, r2, r3;
    unpack2(fma2(pack2(__uint_as_float(hi.x << 16), __uint_as_float(hi.x & 0xffff0000u)), minus, pack2(a, b)), r0, r1);
    unpack2(fma2(pack2(__uint_as_float(hi.y << 16), __uint_as_float(hi.y & 0xffff0000u)), minus, pack2(c, d)), r2, r3);
    lo = make_uint2(cvt_bf16x2(r0, r1), cvt_bf16x2(r2, r3));
}

}  // namespace tc
}  // namespace dpmm
