// The experts' two matrix products for steps of a few dozen to a few hundred tokens, bfloat16, on the fifth-generation tensor
// cores: rows [pairs, K] in the order of their experts (`ends`: each expert's last row + 1, on the device), expert e's
// weight the rows [e w_rows, (e + 1) w_rows) of one matrix.
//
//   kind 0   out[p, :] = rows[p, :] . W_e^T                                     (w_rows = n_out)
//   kind 1   out[p, :] = unit(rows[p, :] . Wg_e^T, rows[p, :] . Wu_e^T)         (w_rows = 2 n_out: gate rows, then up rows)
//   kind 2   out[p, :] = relu(rows[p, :] . W_e^T)^2                             (w_rows = n_out)
//
// Such a step is bound by reading the chosen experts' matrices once.  The operands are swapped, as in the stream-K product: 128
// rows of W (for kind 1 128 gate rows and the 128 up rows that go with them) fill the 128-row side of tcgen05.mma, 32 or 64
// of the expert's rows are the other side.  The items (expert, 128 rows of W, 32 or 64 rows) are counted from `ends` by every
// CTA for itself and walked by one persistent CTA per SM, experts without rows left out; items of one W tile are neighbours, so
// that the second finds W in L2:
//   warp 0, one lane:  TMA into a ring of stages of 64 inputs, on across items without a pause
//   warp 1, one lane:  MMA into one of two sets of accumulators in tensor memory
//   warps 2..5:        epilogue: unit in float32, one rounding, rows beyond the expert's are dropped
// Every wait is bounded: when one runs out a code goes to *error_flag, the roles leave their loops, copies in flight are waited
// for, tensor memory is freed and the kernel returns.
//
// NikolayBlagoev/garlic-inference runs its experts one by one through a library product.
#include "common.cuh"
#include "glu.cuh"

#include <cuda.h>

#define GX_ROWS 128                     // rows of W per tile
#define GX_BK 64
#define GX_THREADS 192
#define GX_W_BYTES (GX_ROWS * GX_BK * 2)
#define GX_MAX_EXPERTS 256
#define GX_SPIN_LIMIT (1 << 22)
#define GX_MAX_STAGES 10

#define GX_ERR_PRODUCER 61
#define GX_ERR_MMA 62
#define GX_ERR_EPILOGUE 63

// Stages that fit one CTA to an SM.
constexpr int gx_stages(int kind, int bn) { return kind == 1 ? (bn == 32 ? 6 : 5) : (bn == 32 ? 10 : 9); }

struct GxControl {
    unsigned long long full[GX_MAX_STAGES], empty[GX_MAX_STAGES];
    unsigned long long acc_full[2], acc_empty[2];
    unsigned int tmem_base;
    int abort;
    int first_item[GX_MAX_EXPERTS + 1];       // items of the experts before
    int first_row[GX_MAX_EXPERTS + 1];        // rows of the experts before
};

__device__ __forceinline__ uint32_t gx_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void gx_mbar_init(void* bar, int count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(gx_smem(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ bool gx_mbar_wait(void* bar, uint32_t parity, volatile int* abort) {
    for (int i = 0; i < GX_SPIN_LIMIT; ++i) {
        uint32_t ok;
        asm volatile("{\n\t.reg .pred p;\n\t"
                     "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                     "selp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(ok) : "r"(gx_smem(bar)), "r"(parity) : "memory");
        if (ok) return true;
        if ((i & 255) == 255 && *abort) return false;
    }
    return false;
}
__device__ __forceinline__ void gx_tma_load_2d(void* dst, const CUtensorMap* map, int x, int y, void* bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
                 ::"r"(gx_smem(dst)), "l"(map), "r"(gx_smem(bar)), "r"(x), "r"(y) : "memory");
}
// K-major tile with rows of 128 bytes, 128-byte swizzle, groups of 8 rows 1,024 bytes apart
__device__ __forceinline__ uint64_t gx_desc(uint32_t addr) {
    return (uint64_t)((addr & 0x3FFFF) >> 4) | (1ull << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
__device__ __forceinline__ void gx_mma(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                 ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void gx_commit(void* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(gx_smem(bar)) : "memory");
}
__device__ __forceinline__ void gx_ld16(uint32_t taddr, float* r) {
    uint32_t u[16];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 "
                 "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                 : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7]),
                   "=r"(u[8]), "=r"(u[9]), "=r"(u[10]), "=r"(u[11]), "=r"(u[12]), "=r"(u[13]), "=r"(u[14]), "=r"(u[15])
                 : "r"(taddr) : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) r[i] = __uint_as_float(u[i]);
}

// What item `t` is: of which expert, which tile of its weight, which of its rows.  `e` goes up with t.
struct GxItem {
    int e, tile, row0, rows;
    __device__ __forceinline__ void at(int t, const GxControl* ctl, int BN) {
        while (t >= ctl->first_item[e + 1]) ++e;
        const int first = ctl->first_row[e], n = ctl->first_row[e + 1] - first;
        const int per = (n + BN - 1) / BN, local = t - ctl->first_item[e];
        tile = local / per;
        const int m = local - tile * per;
        row0 = first + m * BN;
        rows = min(BN, n - m * BN);
    }
};

template <int KIND, int BN>
__global__ void __launch_bounds__(GX_THREADS, 1)
moe_grouped_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, const int* __restrict__ ends,
                   bf16* __restrict__ out, int E, int n_pairs, int n_out, int K, GluShape unit, int* __restrict__ error_flag) {
    constexpr int STAGES = gx_stages(KIND, BN), PARTS = KIND == 1 ? 2 : 1;             // parts: 128-row tiles of W in a stage
    constexpr int X_BYTES = BN * GX_BK * 2, STAGE_BYTES = PARTS * GX_W_BYTES + X_BYTES;
    constexpr int TMEM_COLS = 2 * PARTS * BN;                                          // 64, 128 or 256
    gi_pdl_start();
    extern __shared__ unsigned char gx_raw[];
    unsigned char* smem = (unsigned char*)(((uintptr_t)gx_raw + 1023) & ~(uintptr_t)1023);
    GxControl* ctl = reinterpret_cast<GxControl*>(smem + STAGES * STAGE_BYTES);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, tiles = (n_out + GX_ROWS - 1) / GX_ROWS;
    const int k_blocks = (K + GX_BK - 1) / GX_BK;
    volatile int* abort = &ctl->abort;
    if (warp == 0) {
        // the experts' first rows and items, 32 experts at a time (ends beyond the rows, or falling, count as no rows)
        int items = 0;
        for (int e0 = 0; e0 < E; e0 += 32) {
            const int e = e0 + lane;
            const int hi = e < E ? min(max(ends[e], 0), n_pairs) : 0, lo = e > 0 && e < E ? min(max(ends[e - 1], 0), n_pairs) : 0;
            int mine = e < E ? (max(hi - lo, 0) + BN - 1) / BN * tiles : 0, sum = mine;
            for (int o = 1; o < 32; o <<= 1) {
                const int up = __shfl_up_sync(0xffffffffu, sum, o);
                if (lane >= o) sum += up;
            }
            if (e < E) { ctl->first_item[e] = items + sum - mine; ctl->first_row[e] = lo; ctl->first_row[e + 1] = hi; }
            items += __shfl_sync(0xffffffffu, sum, 31);
            __syncwarp();
        }
        if (lane == 0) {
            ctl->first_item[E] = items;
            for (int s = 0; s < STAGES; ++s) { gx_mbar_init(&ctl->full[s], 1); gx_mbar_init(&ctl->empty[s], 1); }
            for (int b = 0; b < 2; ++b) { gx_mbar_init(&ctl->acc_full[b], 1); gx_mbar_init(&ctl->acc_empty[b], 4); }
            ctl->abort = 0;
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
    } else if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(gx_smem(&ctl->tmem_base)), "r"(TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = ctl->tmem_base;
    const int items = ctl->first_item[E];
    GxItem im;
    im.e = 0;

    if (warp == 0) {
        if (lane == 0) {
            int it = 0;
            bool ok = true;
            for (int t = blockIdx.x; t < items && ok; t += gridDim.x) {
                im.at(t, ctl, BN);
                const int w_row = im.e * (PARTS * n_out) + im.tile * GX_ROWS;
                for (int kb = 0; kb < k_blocks; ++kb, ++it) {
                    const int s = it % STAGES;
                    if (!gx_mbar_wait(&ctl->empty[s], ((it / STAGES) & 1) ^ 1, abort)) {
                        if (!*abort) { *abort = 1; atomicExch(error_flag, GX_ERR_PRODUCER); }
                        ok = false;
                        break;
                    }
                    unsigned char* st = smem + s * STAGE_BYTES;
                    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(gx_smem(&ctl->full[s])), "r"(STAGE_BYTES) : "memory");
                    gx_tma_load_2d(st, &map_w, kb * GX_BK, w_row, &ctl->full[s]);
                    if (PARTS == 2) gx_tma_load_2d(st + GX_W_BYTES, &map_w, kb * GX_BK, w_row + n_out, &ctl->full[s]);
                    gx_tma_load_2d(st + PARTS * GX_W_BYTES, &map_x, kb * GX_BK, im.row0, &ctl->full[s]);
                }
            }
            if (*abort) {                        // let the copies still in flight land before the CTA leaves
                int never = 0;
                for (int i = max(0, it - STAGES); i < it; ++i) gx_mbar_wait(&ctl->full[i % STAGES], (i / STAGES) & 1, &never);
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            // float32 accumulate, bfloat16 operands, both K-major, N = BN, M = 128
            const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(GX_ROWS >> 4) << 24);
            int it = 0, local = 0;
            bool ok = true;
            for (int t = blockIdx.x; t < items && ok; t += gridDim.x, ++local) {
                const int buf = local & 1;
                if (!gx_mbar_wait(&ctl->acc_empty[buf], ((local >> 1) & 1) ^ 1, abort)) {
                    if (!*abort) { *abort = 1; atomicExch(error_flag, GX_ERR_MMA); }
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t acc = tmem + buf * PARTS * BN;
                for (int kb = 0; kb < k_blocks; ++kb, ++it) {
                    const int s = it % STAGES;
                    if (!gx_mbar_wait(&ctl->full[s], (it / STAGES) & 1, abort)) {
                        if (!*abort) { *abort = 1; atomicExch(error_flag, GX_ERR_MMA); }
                        ok = false;
                        break;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t w_addr = gx_smem(smem + s * STAGE_BYTES), x_addr = w_addr + PARTS * GX_W_BYTES;
#pragma unroll
                    for (int k = 0; k < GX_BK / 16; ++k)
#pragma unroll
                        for (int p = 0; p < PARTS; ++p)
                            gx_mma(acc + p * BN, gx_desc(w_addr + p * GX_W_BYTES + k * 32), gx_desc(x_addr + k * 32), idesc, (kb | k) != 0);
                    gx_commit(&ctl->empty[s]);
                }
                if (ok) gx_commit(&ctl->acc_full[buf]);
            }
        }
    } else {
        const int q = warp & 3;
        int local = 0;
        for (int t = blockIdx.x; t < items; t += gridDim.x, ++local) {
            im.at(t, ctl, BN);
            const int buf = local & 1;
            if (!__all_sync(0xffffffffu, gx_mbar_wait(&ctl->acc_full[buf], (local >> 1) & 1, abort))) {
                if (!*abort) { *abort = 1; atomicExch(error_flag, GX_ERR_EPILOGUE); }
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            float v[PARTS][BN];
#pragma unroll
            for (int p = 0; p < PARTS; ++p)
#pragma unroll
                for (int c = 0; c < BN; c += 16) gx_ld16(tmem + ((uint32_t)(q * 32) << 16) + (buf * PARTS + p) * BN + c, &v[p][c]);
            // the accumulators are in registers: the MMA lane may overwrite them
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(gx_smem(&ctl->acc_empty[buf])) : "memory");
            const int col = im.tile * GX_ROWS + q * 32 + lane;
            if (col < n_out) {
                bf16* dst = out + (size_t)im.row0 * n_out + col;
#pragma unroll
                for (int m = 0; m < BN; ++m) {
                    if (m >= im.rows) break;
                    float y = v[0][m];
                    if (KIND == 1) y = glu_unit(y, v[PARTS - 1][m], unit);
                    if (KIND == 2) { y = fmaxf(y, 0.f); y *= y; }
                    dst[(size_t)m * n_out] = __float2bfloat16_rn(y);
                }
            }
            __syncwarp();                        // tensor memory is read by whole warps
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
    }
}

// ------------------------------------------------------------------------------ host side
typedef CUresult (*gx_encode_fn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                 const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                 CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static int gx_make_map(CUtensorMap* map, const void* base, long long rows, int K, int box_rows) {
    static gx_encode_fn enc = nullptr;
    if (!enc) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess)
            enc = (gx_encode_fn)p;
    }
    GI_REQUIRE(enc != nullptr, "gi_moe_grouped: the driver does not offer cuTensorMapEncodeTiled");
    const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)K * 2};
    const cuuint32_t box[2] = {GX_BK, (cuuint32_t)box_rows};
    const cuuint32_t elem[2] = {1, 1};
    CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, elem,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    GI_REQUIRE(r == CUDA_SUCCESS, "gi_moe_grouped: cuTensorMapEncodeTiled failed with code %d", (int)r);
    return 0;
}

template <int KIND, int BN>
static int gx_launch(const void* rows, const void* w, const int* ends, void* out, int E, int n_pairs, int n_out, int K, const GluShape& unit,
                     int* error_flag, cudaStream_t s) {
    CUtensorMap map_w, map_x;
    if (int rc = gx_make_map(&map_w, w, (long long)E * (KIND == 1 ? 2 : 1) * n_out, K, GX_ROWS)) return rc;
    if (int rc = gx_make_map(&map_x, rows, n_pairs, K, BN)) return rc;
    int n_sm = 148, dev = 0;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev);
    const size_t smem = (size_t)gx_stages(KIND, BN) * ((KIND == 1 ? 2 : 1) * GX_W_BYTES + BN * GX_BK * 2) + sizeof(GxControl) + 1024;
    if (int rc = gi_reserve_smem((const void*)moe_grouped_kernel<KIND, BN>, smem, "gi_moe_grouped")) return rc;
    gi_launch(moe_grouped_kernel<KIND, BN>, dim3(n_sm), dim3(GX_THREADS), smem, s, map_w, map_x, ends, (bf16*)out, E, n_pairs, n_out, K, unit,
              error_flag);
    return gi_check_launch("gi_moe_grouped");
}

extern "C" int gi_moe_grouped(const void* rows, const void* w, const int* ends, void* out, int E, int n_pairs, int n_out, int K, int kind,
                              int act, float alpha, float gate_max, float up_limit, float up_shift, int* error_flag, void* stream) {
    GI_REQUIRE(E > 0 && E <= GX_MAX_EXPERTS && n_pairs >= 0 && n_out > 0 && K > 0 && K % 8 == 0, "gi_moe_grouped: %d experts (at most %d), "
               "%d pairs, products of %d x %d (the second a multiple of 8)", E, GX_MAX_EXPERTS, n_pairs, n_out, K);
    GI_REQUIRE(kind >= 0 && kind <= 2, "gi_moe_grouped: kind %d", kind);
    GI_REQUIRE(((uintptr_t)rows | (uintptr_t)w) % 16 == 0 && error_flag != nullptr, "gi_moe_grouped: operands start on 16 bytes; an error flag is required");
    GI_REQUIRE(((long long)n_out + GX_ROWS) / GX_ROWS * ((long long)n_pairs / 32 + E) < (1LL << 31) && (long long)E * 2 * n_out < (1LL << 31),
               "gi_moe_grouped: %d pairs of %d columns", n_pairs, n_out);
    if (n_pairs == 0) return 0;
    const GluShape unit = {act, alpha, gate_max, up_limit, up_shift};
    cudaStream_t s = (cudaStream_t)stream;
    // rows of an expert to an item: 32 while experts have 16 on average (a second item of an expert reads its weight again,
    // out of L2), 64 from there on
    const bool wide = n_pairs > 16 * E;
#define GX_GO(KIND)                                                                                                          \
    return wide ? gx_launch<KIND, 64>(rows, w, ends, out, E, n_pairs, n_out, K, unit, error_flag, s)                         \
                : gx_launch<KIND, 32>(rows, w, ends, out, E, n_pairs, n_out, K, unit, error_flag, s)
    if (kind == 1) GX_GO(1);
    if (kind == 2) GX_GO(2);
    GX_GO(0);
#undef GX_GO
}
