// What kernels on the fifth-generation tensor cores share: mbarriers with bounded waits, tiled TMA loads, matrix
// descriptors, products, tensor memory.
#pragma once
#include "common.cuh"

#include <cuda.h>

#define T5_SPIN_LIMIT (1 << 22)

__device__ __forceinline__ uint32_t t5_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void t5_bar_init(void* bar, int count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(t5_smem(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void t5_bar_expect(void* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(t5_smem(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void t5_bar_arrive(void* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(t5_smem(bar)) : "memory");
}
__device__ __forceinline__ bool t5_bar_try(void* bar, uint32_t parity) {              // may suspend the thread for a while
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\t"
                 "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                 "selp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok) : "r"(t5_smem(bar)), "r"(parity) : "memory");
    return ok != 0;
}
__device__ __forceinline__ bool t5_bar_test(void* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\t"
                 "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                 "selp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok) : "r"(t5_smem(bar)), "r"(parity) : "memory");
    return ok != 0;
}
// Bounded: false when the limit ran out or another role gave up.  What is there already is seen by the first test (75 cycles, a
// try_wait takes 200); who has to wait does so suspended and leaves the issue slots to others.
__device__ __forceinline__ bool t5_bar_wait(void* bar, uint32_t parity, volatile int* abort) {
    if (t5_bar_test(bar, parity)) return true;
    for (int i = 0; i < T5_SPIN_LIMIT; ++i) {
        if (t5_bar_try(bar, parity)) return true;
        if ((i & 255) == 255 && *abort) return false;
    }
    return false;
}
// The same for a whole warp: one lane asks, so that a block's waiting warps leave the barrier unit to the others.  The role
// that gives up first leaves its code.
__device__ __forceinline__ bool t5_warp_wait(void* bar, uint32_t parity, volatile int* abort, int* error_flag, int code) {
    const bool there = (threadIdx.x & 31) != 0 || t5_bar_wait(bar, parity, abort);
    if (__all_sync(0xffffffffu, there)) return true;
    if (!*abort) { *abort = 1; atomicExch(error_flag, code); }
    return false;
}
__device__ __forceinline__ bool t5_lane_wait(void* bar, uint32_t parity, volatile int* abort, int* error_flag, int code) {
    if (t5_bar_wait(bar, parity, abort)) return true;
    if (!*abort) { *abort = 1; atomicExch(error_flag, code); }
    return false;
}
__device__ __forceinline__ void t5_load_2d(void* dst, const CUtensorMap* map, int x, int y, void* bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
                 ::"r"(t5_smem(dst)), "l"(map), "r"(t5_smem(bar)), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ void t5_load_3d(void* dst, const CUtensorMap* map, int x, int y, int z, void* bar) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
                 ::"r"(t5_smem(dst)), "l"(map), "r"(t5_smem(bar)), "r"(x), "r"(y), "r"(z) : "memory");
}
// one lane of a converged warp
__device__ __forceinline__ bool t5_elect() {
    uint32_t chosen;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(chosen));
    return chosen != 0;
}
// Shared-memory descriptor of a K-major tile of rows of ROW bytes (128 or 64) under the swizzle of that width: groups of 8
// rows lie 8 ROW apart.
template <int ROW> __device__ __forceinline__ uint64_t t5_desc(uint32_t addr) {
    static_assert(ROW == 128 || ROW == 64, "rows of one swizzle");
    return (uint64_t)((addr & 0x3FFFF) >> 4) | (1ull << 16) | ((uint64_t)(8 * ROW >> 4) << 32) | (1ull << 46) | ((ROW == 128 ? 2ull : 4ull) << 61);
}
// float32 accumulate, bfloat16 operands, both K-major, M x N
__device__ __forceinline__ constexpr uint32_t t5_idesc(int m, int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}
// the first operand from tensor memory, the second from shared memory
__device__ __forceinline__ void t5_mma_ts(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
                 ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void t5_mma_ss(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                 ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
}
// arrives when the products issued so far are done
__device__ __forceinline__ void t5_commit(void* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(t5_smem(bar)) : "memory");
}
__device__ __forceinline__ void t5_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void t5_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void t5_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void t5_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// whole warps; `where` is shared memory that gets the address
__device__ __forceinline__ void t5_alloc(void* where, int columns) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(t5_smem(where)), "r"(columns) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void t5_free(uint32_t tmem, int columns) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(columns) : "memory");
}
// a lane's row of N columns (the caller waits)
template <int N> __device__ __forceinline__ void t5_ld(uint32_t at, float (&r)[N]) {
    static_assert(N == 8 || N == 16 || N == 32, "columns of one load");
    if constexpr (N == 8)
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                     : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]), "=f"(r[4]), "=f"(r[5]), "=f"(r[6]), "=f"(r[7]) : "r"(at) : "memory");
    else if constexpr (N == 16)
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                     : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]), "=f"(r[4]), "=f"(r[5]), "=f"(r[6]), "=f"(r[7]),
                       "=f"(r[8]), "=f"(r[9]), "=f"(r[10]), "=f"(r[11]), "=f"(r[12]), "=f"(r[13]), "=f"(r[14]), "=f"(r[15])
                     : "r"(at) : "memory");
    else
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 "
                     "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
                     "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
                     : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]), "=f"(r[4]), "=f"(r[5]), "=f"(r[6]), "=f"(r[7]),
                       "=f"(r[8]), "=f"(r[9]), "=f"(r[10]), "=f"(r[11]), "=f"(r[12]), "=f"(r[13]), "=f"(r[14]), "=f"(r[15]),
                       "=f"(r[16]), "=f"(r[17]), "=f"(r[18]), "=f"(r[19]), "=f"(r[20]), "=f"(r[21]), "=f"(r[22]), "=f"(r[23]),
                       "=f"(r[24]), "=f"(r[25]), "=f"(r[26]), "=f"(r[27]), "=f"(r[28]), "=f"(r[29]), "=f"(r[30]), "=f"(r[31])
                     : "r"(at) : "memory");
}
__device__ __forceinline__ void t5_st8(uint32_t at, const uint32_t (&r)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                 ::"r"(at), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
}
__device__ __forceinline__ void t5_st16(uint32_t at, const uint32_t (&r)[16]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
                 ::"r"(at), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
                   "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]) : "memory");
}

// {x, y} as three pairs of bfloat16 that sum to them exactly: each part is what is left, rounded to nearest, so that a part is at most
// 2^-9 of the one before it (24 bits of mantissa = 8 + 8 + 8).  Not for infinities, NaN and what rounds to an infinity, and below 2^-110 only to
// 2^-134, half of bfloat16's smallest number.
typedef unsigned long long t5_f2;             // two floats in a register pair
__device__ __forceinline__ t5_f2 t5_pair(float x, float y) {
    t5_f2 d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(x), "f"(y));
    return d;
}
__device__ __forceinline__ void t5_apart(t5_f2 v, float& x, float& y) { asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(v)); }
__device__ __forceinline__ t5_f2 t5_add2(t5_f2 a, t5_f2 b) {
    t5_f2 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ t5_f2 t5_mul2(t5_f2 a, t5_f2 b) {
    t5_f2 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ t5_f2 t5_fma2(t5_f2 a, t5_f2 b, t5_f2 c) {
    t5_f2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ void t5_split3(float x, float y, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
    const t5_f2 minus = t5_pair(-1.f, -1.f);
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(hi) : "f"(y), "f"(x));
    t5_f2 r = t5_fma2(t5_pair(__uint_as_float(hi << 16), __uint_as_float(hi & 0xffff0000u)), minus, t5_pair(x, y));
    float rx, ry;
    t5_apart(r, rx, ry);
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(mid) : "f"(ry), "f"(rx));
    r = t5_fma2(t5_pair(__uint_as_float(mid << 16), __uint_as_float(mid & 0xffff0000u)), minus, r);
    t5_apart(r, rx, ry);
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(lo) : "f"(ry), "f"(rx));
}

// Host: a [rows, cols] row-major matrix, rows `stride` bytes apart, as a 2-D map with boxes of box_rows x (one swizzle width) and zeros
// outside; with `planes`, that many such matrices one behind the other as a 3-D map whose boxes take all of them.  0 or an error code
// (gi_last_error names `who`).
int t5_make_map(CUtensorMap* map, CUtensorMapDataType type, int elem_bytes, const void* base, long long rows, long long cols, long long stride,
                int box_rows, int box_cols, CUtensorMapSwizzle swizzle, const char* who, int planes = 0);
