// The gates of the real-gated linear recurrent unit (rglru.cu) over many rows, for bfloat16 matrices, on the fifth-generation tensor
// cores:  a = exp(-c sigmoid(Wa u + ba) softplus(lam)),  b = sqrt(1 - a^2) sigmoid(Wi u + bi) u  per block of channels.
//
// 128 rows of u are the wide side; the other are 64 outputs of both gates.  A float32 input is the exact sum of three bfloat16 numbers,
// and every product of one of them with a weight is exact in float32.  The accumulator starts from zero for every 64 inputs and
// takes the products of the third parts first, of the first parts last; these sums meet in registers by float32 adds that round
// to nearest (the tensor core cuts its sums off, which is why they are kept short).
//   warps 0..3     split u: TMA brings 128 rows x 64 inputs, a lane takes a row and puts its parts into tensor memory
//   warps 4..19    add the sums up and make a and b from them: four groups of four, 16 outputs of both gates each
//   warps 20..22   TMA of u, TMA of both matrices, products
// Bound by what is done one after another for an item: products, sums and then some 100 instructions for an output, while all adders wait
// for one item at a time.  At 16 blocks of 320 the tensor core is busy for 16 % of the time, the issue slots for 56 %.
// Measured, 16 blocks of 320, 2,494 rows: 213 us by mma.sync (rglru.cu: three legacy products and four adds for every 16 inputs, and 250
// instructions an output), 192 us so, 138 us with the divisions and roots below.  Relative errors of b (2-norm) against 64 bits in
// units of 1e-8, mma.sync / so: blocks of 64 7.4 / 7.5, 72 7.6 / 7.6, 320 8.0 / 7.8, 1,280 9.6 / 8.3; inputs of three times the size 8.9 / 8.4;
// a's 3.2 / 3.2.
#include "rglru.cuh"
#include "tcgen05.cuh"

#define RT_ROWS 128
#define RT_OUT 64                    // outputs of each gate to an item
#define RT_BK 64                     // inputs to a slice and to a sum
#define RT_U_BYTES (RT_ROWS * RT_BK * 4)
#define RT_W_BYTES (2 * RT_OUT * RT_BK * 2)
#define RT_US 3
#define RT_WS 6
#define RT_RING 8
#define RT_ACCS 2
#define RT_SPLITS 2
#define RT_COLS (2 * RT_OUT)         // columns of an accumulator
#define RT_A_COLS (3 * RT_BK / 2)    // of a split slice
#define RT_ADDERS 16
#define RT_THREADS ((4 + RT_ADDERS + 3) * 32)
#define RT_SMEM (RT_US * RT_U_BYTES + RT_WS * RT_W_BYTES + sizeof(RtControl) + 1024)

#define RT_ERR_COPY 91
#define RT_ERR_SPLIT 92
#define RT_ERR_MMA 93
#define RT_ERR_ADD 94

struct RtControl {
    unsigned long long u_full[RT_RING], u_empty[RT_RING], w_full[RT_RING], split[RT_RING], done[RT_RING], acc_full[RT_ACCS], acc_empty[RT_ACCS];
    unsigned int tmem_base;
    int abort;
};

struct Floats8 { float v[8]; };      // 32 bytes: a whole sector a lane
__device__ __forceinline__ Floats8 rt_load8(const float* p) {
    Floats8 r;
    asm volatile("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=f"(r.v[0]), "=f"(r.v[1]), "=f"(r.v[2]), "=f"(r.v[3]), "=f"(r.v[4]), "=f"(r.v[5]), "=f"(r.v[6]), "=f"(r.v[7]) : "l"(p));
    return r;
}
__device__ __forceinline__ void rt_store8(float* p, const Floats8& r) {
    asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                 ::"l"(p), "f"(r.v[0]), "f"(r.v[1]), "f"(r.v[2]), "f"(r.v[3]), "f"(r.v[4]), "f"(r.v[5]), "f"(r.v[6]), "f"(r.v[7]) : "memory");
}

// 1 / (1 + exp(-z)): the hardware's reciprocal and one step of Newton's method, x (2 - d x), without the branches of a division
__device__ __forceinline__ float rt_sigmoid(float z) {
    const float d = 1.f + expf(-z);
    float x;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(x) : "f"(d));
    x = fmaf(x, fmaf(-d, x, 1.f), x);
    return d < 1e37f ? x : d != d ? d : 0.f;                 // (beyond, the step would multiply zero by infinity)
}
// sqrt(1 - exp(y)) for y <= 0.  1 - exp(y) keeps its digits where y is small by Taylor's series of (exp(y) - 1) / y around zero, whose
// first dropped term is 1 / 12! there; the root by the hardware's reciprocal root and one step of Newton's method.
__device__ __forceinline__ float rt_keep(float y) {
    float t = 1.f / 39916800.f;
    t = fmaf(t, y, 1.f / 3628800.f);
    t = fmaf(t, y, 1.f / 362880.f);
    t = fmaf(t, y, 1.f / 40320.f);
    t = fmaf(t, y, 1.f / 5040.f);
    t = fmaf(t, y, 1.f / 720.f);
    t = fmaf(t, y, 1.f / 120.f);
    t = fmaf(t, y, 1.f / 24.f);
    t = fmaf(t, y, 1.f / 6.f);
    t = fmaf(t, y, 0.5f);
    t = fmaf(t * y, y, y);
    const float x = y > -1.f ? -t : 1.f - expf(y);
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    const float s = x * r;
    return x > 1.2e-38f ? fmaf(fmaf(-s, s, x), 0.5f * r, s) : sqrtf(fmaxf(x, 0.f));
}

__global__ void __launch_bounds__(RT_THREADS, 1)
rglru_gates_tcgen05_kernel(const __grid_constant__ CUtensorMap map_u, const __grid_constant__ CUtensorMap map_wa,
                           const __grid_constant__ CUtensorMap map_wi, const float* __restrict__ u, const bf16* __restrict__ wa_t,
                           const bf16* __restrict__ wi_t, const void* __restrict__ ba, const void* __restrict__ bi, const void* __restrict__ lam,
                           int vec_dtype, float decay_scale, float* __restrict__ a_out, float* __restrict__ b_out, int n_rows, int width,
                           int blocks, int bw, int* __restrict__ error_flag) {
    gi_pdl_launch_dependents();
    extern __shared__ unsigned char rt_raw[];
    unsigned char* smem = (unsigned char*)(((uintptr_t)rt_raw + 1023) & ~(uintptr_t)1023);
    unsigned char* w_tiles = smem + RT_US * RT_U_BYTES;
    RtControl* ctl = reinterpret_cast<RtControl*>(w_tiles + RT_WS * RT_W_BYTES);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // item: (tile of rows, block of channels, 64 of its outputs), outputs fastest
    const int outs = (bw + RT_OUT - 1) / RT_OUT, items = (n_rows + RT_ROWS - 1) / RT_ROWS * blocks * outs, slices = (bw + RT_BK - 1) / RT_BK;
    const int own = ((int)blockIdx.x < items ? (items - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0) * slices;
    volatile int* abort = &ctl->abort;

    if (threadIdx.x == 0) {
        for (int s = 0; s < RT_RING; ++s) {
            t5_bar_init(&ctl->u_full[s], 1); t5_bar_init(&ctl->u_empty[s], 4); t5_bar_init(&ctl->w_full[s], 1);
            t5_bar_init(&ctl->split[s], 4); t5_bar_init(&ctl->done[s], 1);
        }
        for (int s = 0; s < RT_ACCS; ++s) { t5_bar_init(&ctl->acc_full[s], 1); t5_bar_init(&ctl->acc_empty[s], RT_ADDERS); }
        ctl->abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 22) t5_alloc(&ctl->tmem_base, 512);
    t5_fence_before();
    __syncthreads();
    t5_fence_after();
    const uint32_t tmem = ctl->tmem_base, split0 = tmem + RT_ACCS * RT_COLS;

    if (warp < 4) {
        gi_pdl_wait();
        const int row = warp * 32 + lane, swap = row & 7;
        for (int it = 0; it < own; ++it) {
            const int s = it % RT_US, last = it - RT_SPLITS;                // the slice that had these columns before
            const uint32_t at = split0 + it % RT_SPLITS * RT_A_COLS + ((uint32_t)(warp * 32) << 16);
            if (!t5_warp_wait(&ctl->u_full[s], it / RT_US & 1, abort, error_flag, RT_ERR_SPLIT)) break;
            if (last >= 0 && !t5_warp_wait(&ctl->done[last % RT_RING], last / RT_RING & 1, abort, error_flag, RT_ERR_SPLIT)) break;
            t5_fence_after();
#pragma unroll
            for (int c = 0; c < RT_BK / 16; ++c) {           // 16 inputs at a time, as the 128-byte swizzle put them
                const unsigned char* src = smem + s * RT_U_BYTES + (c >> 1) * (RT_U_BYTES / 2) + row * 128;
                uint32_t part[3][8];
#pragma unroll
                for (int w = 0; w < 4; ++w) {
                    const float4 v = *reinterpret_cast<const float4*>(src + ((((c & 1) * 4 + w) ^ swap) << 4));
                    t5_split3(v.x, v.y, part[0][2 * w], part[1][2 * w], part[2][2 * w]);
                    t5_split3(v.z, v.w, part[0][2 * w + 1], part[1][2 * w + 1], part[2][2 * w + 1]);
                }
#pragma unroll
                for (int p = 0; p < 3; ++p) t5_st8(at + p * (RT_BK / 2) + c * 8, part[p]);
            }
            t5_wait_st();
            t5_fence_before();
            __syncwarp();
            if (lane == 0) {
                t5_bar_arrive(&ctl->split[it % RT_RING]);
                t5_bar_arrive(&ctl->u_empty[s]);
            }
        }
    } else if (warp < 4 + RT_ADDERS) {
        gi_pdl_wait();
        const int q = warp & 3, group = (warp - 4) >> 2;
        const uint32_t at = tmem + ((uint32_t)(q * 32) << 16) + group * 16;
        int it = 0;
        bool ok = true;
        for (int item = blockIdx.x; item < items && ok; item += gridDim.x) {
            const int o0 = item % outs * RT_OUT + group * 16, blk = item / outs % blocks, row = item / outs / blocks * RT_ROWS + q * 32 + lane;
            // lane l keeps what output l of the 16 needs: both biases and softplus(lam)
            const int ch = blk * bw + min(o0 + (lane & 15), bw - 1);
            const float vba = load_w(ba, vec_dtype, ch), vbi = load_w(bi, vec_dtype, ch), vsp = rg_softplus(load_w(lam, vec_dtype, ch));
            t5_f2 za[8], zi[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) za[i] = zi[i] = 0ull;
            for (int k = 0; k < slices; ++k, ++it) {
                const int b = it % RT_ACCS;
                if (!t5_warp_wait(&ctl->acc_full[b], it / RT_ACCS & 1, abort, error_flag, RT_ERR_ADD)) { ok = false; break; }
                t5_fence_after();
                float x[16], y[16];
                t5_ld<16>(at + b * RT_COLS, x);
                t5_ld<16>(at + b * RT_COLS + RT_OUT, y);
                t5_wait_ld();
                t5_fence_before();
                __syncwarp();
                if (lane == 0) t5_bar_arrive(&ctl->acc_empty[b]);
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    za[i] = t5_add2(za[i], t5_pair(x[2 * i], x[2 * i + 1]));
                    zi[i] = t5_add2(zi[i], t5_pair(y[2 * i], y[2 * i + 1]));
                }
            }
            if (!ok) break;
            const size_t first = (size_t)min(row, n_rows - 1) * width + blk * bw;
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                if (o0 + half * 8 < bw) {                    // (the same for the whole warp; bw is a multiple of 8)
                    const Floats8 x = rt_load8(u + first + o0 + half * 8);
                    Floats8 ra, rb;
#pragma unroll
                    for (int e = 0; e < 8; ++e) {
                        float pa[2], pi[2];
                        t5_apart(za[half * 4 + e / 2], pa[0], pa[1]);
                        t5_apart(zi[half * 4 + e / 2], pi[0], pi[1]);
                        float a = pa[e & 1], i = pi[e & 1];
                        if (a != a || i != i) {              // an infinity among the inputs or weights, or a NaN
                            a = rm_plain(u + first, wa_t + (size_t)blk * bw * bw + o0 + half * 8 + e, bw);
                            i = rm_plain(u + first, wi_t + (size_t)blk * bw * bw + o0 + half * 8 + e, bw);
                        }
                        const float r = rt_sigmoid(a + __shfl_sync(0xffffffffu, vba, half * 8 + e));
                        const float g = rt_sigmoid(i + __shfl_sync(0xffffffffu, vbi, half * 8 + e));
                        const float log_a = -decay_scale * r * __shfl_sync(0xffffffffu, vsp, half * 8 + e);
                        ra.v[e] = expf(log_a);
                        rb.v[e] = rt_keep(2.f * log_a) * g * x.v[e];
                    }
                    if (row < n_rows) {
                        rt_store8(a_out + first + o0 + half * 8, ra);
                        rt_store8(b_out + first + o0 + half * 8, rb);
                    }
                }
            }
        }
    } else if (warp < 22) {
        if (lane == 0) {
            // the matrices are nobody's output: their first slices are asked for before the kernel that makes u has finished
            const bool of_u = warp == 20;
            if (of_u) gi_pdl_wait();
            const int ring = of_u ? RT_US : RT_WS;
            int item = blockIdx.x, k = 0, armed = 0;
            for (int it = 0, s = 0, turn = 0; it < own; ++it) {
                const int last = it - RT_WS;
                if (of_u ? turn > 0 && !t5_lane_wait(&ctl->u_empty[s], (turn & 1) ^ 1, abort, error_flag, RT_ERR_COPY)
                         : last >= 0 && !t5_lane_wait(&ctl->done[last % RT_RING], last / RT_RING & 1, abort, error_flag, RT_ERR_COPY)) break;
                const int blk = item / outs % blocks;
                if (of_u) {
                    const int y = item / outs / blocks * RT_ROWS;
                    t5_bar_expect(&ctl->u_full[s], RT_U_BYTES);
                    t5_load_2d(smem + s * RT_U_BYTES, &map_u, blk * bw + k, y, &ctl->u_full[s]);
                    t5_load_2d(smem + s * RT_U_BYTES + RT_U_BYTES / 2, &map_u, blk * bw + k + RT_BK / 2, y, &ctl->u_full[s]);
                } else {
                    const int y = blk * bw + item % outs * RT_OUT;
                    t5_bar_expect(&ctl->w_full[s], RT_W_BYTES);
                    t5_load_2d(w_tiles + s * RT_W_BYTES, &map_wa, k, y, &ctl->w_full[s]);
                    t5_load_2d(w_tiles + s * RT_W_BYTES + RT_W_BYTES / 2, &map_wi, k, y, &ctl->w_full[s]);
                }
                armed = it + 1;
                if (++s == ring) { s = 0; ++turn; }
                if ((k += RT_BK) >= bw) { k = 0; item += gridDim.x; }
            }
            if (!of_u) gi_pdl_wait();
            if (*abort) {                                    // the copies still in flight land before the block leaves
                int never = 0;
                for (int i = max(0, armed - ring); i < armed; ++i) t5_bar_wait(of_u ? &ctl->u_full[i % ring] : &ctl->w_full[i % ring], i / ring & 1, &never);
            }
        }
    } else {
        const bool chosen = t5_elect();
        constexpr uint32_t idesc = t5_idesc(RT_ROWS, RT_COLS);
        for (int it = 0; it < own; ++it) {
            const int b = it % RT_ACCS;
            if (!t5_warp_wait(&ctl->acc_empty[b], (it / RT_ACCS & 1) ^ 1, abort, error_flag, RT_ERR_MMA)) break;
            if (!t5_warp_wait(&ctl->w_full[it % RT_WS], it / RT_WS & 1, abort, error_flag, RT_ERR_MMA)) break;
            if (!t5_warp_wait(&ctl->split[it % RT_RING], it / RT_RING & 1, abort, error_flag, RT_ERR_MMA)) break;
            t5_fence_after();
            const uint32_t d = tmem + b * RT_COLS, parts = split0 + it % RT_SPLITS * RT_A_COLS;
            const uint64_t w = t5_desc<128>(t5_smem(w_tiles + it % RT_WS * RT_W_BYTES));
            if (chosen) {
#pragma unroll
                for (int p = 2; p >= 0; --p)
#pragma unroll
                    for (int k = 0; k < RT_BK / 16; ++k)     // 16 inputs: 8 columns of tensor memory, 32 bytes of a row of weights
                        t5_mma_ts(d, parts + p * (RT_BK / 2) + k * 8, w + k * 2, idesc, p != 2 || k);
                t5_commit(&ctl->done[it % RT_RING]);
                t5_commit(&ctl->acc_full[b]);
            }
            __syncwarp();
        }
    }
    t5_fence_before();
    __syncthreads();
    if (warp == 22) {
        t5_fence_after();
        t5_free(tmem, 512);
    }
}

// The arguments of gi_rglru_gates, the matrices also as [blocks, out, in]; blocks of a multiple of 8 channels, u, a and b on 32 bytes.
extern "C" int gi_rglru_gates_tcgen05(const float* u, const void* wa, const void* wi, const void* wa_t, const void* wi_t, const void* ba, const void* bi,
                                      const void* lam, int vec_dtype, float decay_scale, float* a_out, float* b_out, int n_rows, int width,
                                      int blocks, int* error_flag, void* stream) {
    GI_REQUIRE(n_rows >= 0 && width > 0 && blocks > 0 && width % blocks == 0, "gi_rglru_gates_tcgen05: %d channels in %d blocks", width, blocks);
    const int bw = width / blocks;
    GI_REQUIRE(bw % 8 == 0 && ((uintptr_t)u | (uintptr_t)a_out | (uintptr_t)b_out) % 32 == 0, "gi_rglru_gates_tcgen05: blocks of %d channels, rows on 32 bytes", bw);
    GI_REQUIRE(error_flag != nullptr, "gi_rglru_gates_tcgen05: an error flag on the device is required");
    const long long items = (long long)((n_rows + RT_ROWS - 1) / RT_ROWS) * blocks * ((bw + RT_OUT - 1) / RT_OUT);
    GI_REQUIRE(items * ((bw + RT_BK - 1) / RT_BK) < 1 << 30, "gi_rglru_gates_tcgen05: %d rows of %d channels", n_rows, width);
    if (n_rows == 0) return 0;
    int n_sm = 148, dev = 0;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev);
    const char* who = "gi_rglru_gates_tcgen05";
    CUtensorMap map_u, map_wa, map_wi;
    if (int rc = t5_make_map(&map_u, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, u, n_rows, width, width * 4LL, RT_ROWS, RT_BK / 2, CU_TENSOR_MAP_SWIZZLE_128B, who)) return rc;
    if (int rc = t5_make_map(&map_wa, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, wa, width, bw, bw * 2LL, RT_OUT, RT_BK, CU_TENSOR_MAP_SWIZZLE_128B, who)) return rc;
    if (int rc = t5_make_map(&map_wi, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, wi, width, bw, bw * 2LL, RT_OUT, RT_BK, CU_TENSOR_MAP_SWIZZLE_128B, who)) return rc;
    if (int rc = gi_reserve_smem((const void*)rglru_gates_tcgen05_kernel, RT_SMEM, who)) return rc;
    gi_launch(rglru_gates_tcgen05_kernel, dim3((unsigned)(items < n_sm ? items : n_sm)), dim3(RT_THREADS), RT_SMEM, (cudaStream_t)stream, map_u, map_wa,
              map_wi, u, (const bf16*)wa_t, (const bf16*)wi_t, ba, bi, lam, vec_dtype, decay_scale, a_out, b_out, n_rows, width, blocks, bw, error_flag);
    return gi_check_launch(who);
}
