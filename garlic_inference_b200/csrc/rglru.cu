// The real-gated linear recurrent unit: a recurrence with one number of state per channel, whose decay and input
// gate are made from the recurrence's own input by block-diagonal matrices.
//
//   gi_rglru_gates   per token, for channels in `blocks` equal blocks:  r = sigmoid(Wa[b] u_b + ba),
//                    i = sigmoid(Wi[b] u_b + bi);  log a = -c r softplus(lam);  a = exp(log a);
//                    b = sqrt(1 - a^2) i u.   Writes a and b as float32 [n, width].  u is float32 (the output of the
//                    short convolution).  1 - a^2 is taken as -expm1(2 log a), which keeps its digits when a is
//                    close to 1.
//   gi_rglru_scan    S_t = a_t S_(t-1) + b_t per channel along each sequence's rows of the step, from the slot's
//                    state row (float32, zero for a new sequence) and back into it; out = S_t * act(y_t + by)
//                    with act the tanh form of gelu, rounded once into the activation type.
//
// The gate matrices arrive transposed, [blocks, in, out]; a block of threads keeps a slice of output channels of
// both matrices in shared memory and streams tiles of tokens past them.  In this file every sum runs in an order that depends on
// the block width alone, and the scan walks a sequence's tokens in order: in the 32-bit engine a position's bits do not depend on
// how the tokens were cut into steps or on the batch.  In bfloat16 steps of many rows have their gates from rglru_tcgen05.cu, as
// precise but with other bits, so there they follow the step's row count.  NikolayBlagoev/garlic-inference has no recurrent mixer.
#include "rglru.cuh"

#define RG_KS 8              // lanes that share an output: lane s sums the inputs k = s, s + 8, s + 16, ...
#define RG_TG 8              // tokens per thread
#define RG_OG 4              // outputs per thread
#define RG_WPAD 8            // padding of a row of weights in shared memory: rows start on 16 bytes and spread over the banks

__device__ __forceinline__ float rg_gelu_tanh(float z) {
    return 0.5f * z * (1.f + tanhf(0.7978845608028654f * (z + 0.044715f * z * z * z)));
}

__device__ __forceinline__ void rg_cp_async_4(float* smem, const float* gmem) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(gmem));
}
__device__ __forceinline__ void rg_cp_async_16(void* smem, const void* gmem, int bytes) {      // the rest of the 16 is zero-filled
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(gmem), "r"(bytes));
}
// 4 bytes, the first n of them copied and the others zero
__device__ __forceinline__ void rg_cp_async_4n(void* dst, const void* src, int n) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(n));
}
__device__ __forceinline__ void rg_cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
__device__ __forceinline__ void rg_cp_async_wait_1() { asm volatile("cp.async.wait_group 1;\n" ::); }
__device__ __forceinline__ void rg_cp_async_wait_0() { asm volatile("cp.async.wait_group 0;\n" ::); }

template <typename TW> __device__ __forceinline__ void rg_load4(const TW* p, float (&w)[4]);
template <> __device__ __forceinline__ void rg_load4<float>(const float* p, float (&w)[4]) {
    const float4 v = *reinterpret_cast<const float4*>(p);
    w[0] = v.x; w[1] = v.y; w[2] = v.z; w[3] = v.w;
}
template <> __device__ __forceinline__ void rg_load4<bf16>(const bf16* p, float (&w)[4]) {
    const uint2 v = *reinterpret_cast<const uint2*>(p);
    const float2 lo = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&v.x));
    const float2 hi = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&v.y));
    w[0] = lo.x; w[1] = lo.y; w[2] = hi.x; w[3] = hi.y;
}

// One block of threads owns `orange` output channels of one block of channels: it copies their two slices of
// the gate matrices into shared memory once ([gate][input][output], rows padded by 8 elements) and then walks its
// share of the step's rows in tiles of `tt` tokens, whose inputs lie in shared memory transposed ([input][token],
// rows padded by 4 floats; two tiles, the next one copied in while this one is summed).  A thread holds 8 tokens x 4 outputs x 2 gates; the 8 lanes that share those outputs
// each sum every eighth input in rising order and their sums meet in a fixed butterfly, so a token's bits depend
// neither on the tile nor on the step's other rows.  The same launch shape serves a prompt (weights read once per
// block of threads, all tokens streamed past them) and a decode step (the weights land in shared memory with
// coalesced loads instead of a chain of dependent ones).
template <typename TW>
__global__ void __launch_bounds__(256)
rglru_gates_kernel(const float* __restrict__ u, const TW* __restrict__ wa_t, const TW* __restrict__ wi_t,
                   const void* __restrict__ ba, const void* __restrict__ bi, const void* __restrict__ lam, int vec_dtype,
                   float decay_scale, float* __restrict__ a_out, float* __restrict__ b_out, int n_rows, int width,
                   int bw, int orange, int tt, int rows_per_cta) {
    gi_pdl_start();
    extern __shared__ __align__(16) unsigned char rg_smem[];
    const int ws = orange + RG_WPAD, us_ld = tt + 4;
    TW* w_s = reinterpret_cast<TW*>(rg_smem);                                     // [2][bw][ws]
    float* u_s = reinterpret_cast<float*>(rg_smem + (((size_t)2 * bw * ws * sizeof(TW) + 15) & ~(size_t)15));   // [2][bw][us_ld]
    const int blk = blockIdx.x, o0 = blockIdx.y * orange;
    const int row_begin = blockIdx.z * rows_per_cta, row_end = min(n_rows, row_begin + rows_per_cta);
    if (row_begin >= row_end) return;
    // the two slices of weights: 16 bytes at a time and asynchronously where rows and slices start on 16 bytes (the
    // part of a chunk beyond the block's last output is zero-filled), element by element otherwise
    constexpr int EPC = 16 / (int)sizeof(TW);               // elements per chunk
    const bool wide = (bw % EPC == 0) && ((uintptr_t)wa_t % 16 == 0) && ((uintptr_t)wi_t % 16 == 0);
    for (int g = 0; g < 2; ++g) {
        const TW* src = (g ? wi_t : wa_t) + (size_t)blk * bw * bw;
        TW* dst = w_s + (size_t)g * bw * ws;
        if (wide) {
            const int cpr = orange / EPC, shift = __ffs(cpr) - 1;          // chunks per row: a power of two
            for (int i = threadIdx.x; i < bw * cpr; i += blockDim.x) {
                const int k = i >> shift, c = i & (cpr - 1), o = o0 + c * EPC;
                const int valid = max(0, min(EPC, bw - o)) * (int)sizeof(TW);
                rg_cp_async_16(dst + (size_t)k * ws + c * EPC, src + (size_t)k * bw + (valid ? o : 0), valid);
            }
        } else {
            for (int k = 0; k < bw; ++k)
                for (int oo = threadIdx.x; oo < orange; oo += blockDim.x)
                    dst[(size_t)k * ws + oo] = o0 + oo < bw ? src[(size_t)k * bw + o0 + oo] : from_f32<TW>(0.f);
        }
    }
    const int n_og = orange / RG_OG;
    const int ks = threadIdx.x % RG_KS, og = (threadIdx.x / RG_KS) % n_og, tg = threadIdx.x / (RG_KS * n_og);
    const int oo = og * RG_OG;                               // first of this thread's outputs within the slice
    // what the epilogue needs of this thread's outputs: biases and softplus(lam)
    float bra[RG_OG], bri[RG_OG], sp[RG_OG];
#pragma unroll
    for (int j = 0; j < RG_OG; ++j) {
        const int o = o0 + oo + j, c = blk * bw + min(o, bw - 1);
        bra[j] = load_w(ba, vec_dtype, c);
        bri[j] = load_w(bi, vec_dtype, c);
        sp[j] = rg_softplus(load_w(lam, vec_dtype, c));
    }
    // A tile's inputs go from global memory straight into their transposed places, four bytes at a time and
    // asynchronously; the tile after the present one is on its way while this one is summed.
    auto issue_tile = [&](int tile0, float* dst) {
        for (int t = 0; t < tt; ++t) {
            const int row = tile0 + t;
            if (row < row_end) {
                const float* src = u + (size_t)row * width + blk * bw;
                for (int k = threadIdx.x; k < bw; k += blockDim.x) rg_cp_async_4(dst + k * us_ld + t, src + k);
            } else {
                for (int k = threadIdx.x; k < bw; k += blockDim.x) dst[k * us_ld + t] = 0.f;
            }
        }
    };
    issue_tile(row_begin, u_s);
    rg_cp_async_commit();
    int it = 0;
    for (int tile0 = row_begin; tile0 < row_end; tile0 += tt, ++it) {
        const float* cur = u_s + (size_t)(it & 1) * bw * us_ld;
        if (tile0 + tt < row_end) issue_tile(tile0 + tt, u_s + (size_t)((it + 1) & 1) * bw * us_ld);
        rg_cp_async_commit();                                // an empty group when nothing is left: the count stays uniform
        rg_cp_async_wait_1();
        __syncthreads();                                     // every thread's copies of this tile have landed (and the weights)
        float ra[RG_TG][RG_OG], ri[RG_TG][RG_OG];
#pragma unroll
        for (int t = 0; t < RG_TG; ++t)
#pragma unroll
            for (int j = 0; j < RG_OG; ++j) ra[t][j] = ri[t][j] = 0.f;
#pragma unroll 2
        for (int k = ks; k < bw; k += RG_KS) {
            float wa4[4], wi4[4];
            rg_load4<TW>(w_s + (size_t)k * ws + oo, wa4);
            rg_load4<TW>(w_s + ((size_t)bw + k) * ws + oo, wi4);
            const float4 x0 = *reinterpret_cast<const float4*>(cur + k * us_ld + tg * RG_TG);
            const float4 x1 = *reinterpret_cast<const float4*>(cur + k * us_ld + tg * RG_TG + 4);
            const float x[RG_TG] = {x0.x, x0.y, x0.z, x0.w, x1.x, x1.y, x1.z, x1.w};
#pragma unroll
            for (int t = 0; t < RG_TG; ++t)
#pragma unroll
                for (int j = 0; j < RG_OG; ++j) {
                    ra[t][j] = fmaf(wa4[j], x[t], ra[t][j]);
                    ri[t][j] = fmaf(wi4[j], x[t], ri[t][j]);
                }
        }
        // The 8 lanes' sums meet in a butterfly that also shares the tokens out: after the exchange with lane s ^ 4
        // a lane keeps the half of its tokens that its bit 2 names, then the quarter its bit 1 names, then one:
        // lane s ends with token s, summed as ((s0 + s4) + (s2 + s6)) + ((s1 + s5) + (s3 + s7)) for every token
        // (the pairs are the same whichever lane keeps the sum), with 56 exchanges instead of 192.
        const bool b2 = ks & 4, b1 = ks & 2, b0 = ks & 1;
        float a4[4][RG_OG], i4[4][RG_OG], a2[2][RG_OG], i2[2][RG_OG], a1[RG_OG], i1[RG_OG];
#pragma unroll
        for (int t = 0; t < 4; ++t)
#pragma unroll
            for (int j = 0; j < RG_OG; ++j) {
                a4[t][j] = (b2 ? ra[t + 4][j] : ra[t][j]) + __shfl_xor_sync(0xffffffffu, b2 ? ra[t][j] : ra[t + 4][j], 4);
                i4[t][j] = (b2 ? ri[t + 4][j] : ri[t][j]) + __shfl_xor_sync(0xffffffffu, b2 ? ri[t][j] : ri[t + 4][j], 4);
            }
#pragma unroll
        for (int t = 0; t < 2; ++t)
#pragma unroll
            for (int j = 0; j < RG_OG; ++j) {
                a2[t][j] = (b1 ? a4[t + 2][j] : a4[t][j]) + __shfl_xor_sync(0xffffffffu, b1 ? a4[t][j] : a4[t + 2][j], 2);
                i2[t][j] = (b1 ? i4[t + 2][j] : i4[t][j]) + __shfl_xor_sync(0xffffffffu, b1 ? i4[t][j] : i4[t + 2][j], 2);
            }
#pragma unroll
        for (int j = 0; j < RG_OG; ++j) {
            a1[j] = (b0 ? a2[1][j] : a2[0][j]) + __shfl_xor_sync(0xffffffffu, b0 ? a2[0][j] : a2[1][j], 1);
            i1[j] = (b0 ? i2[1][j] : i2[0][j]) + __shfl_xor_sync(0xffffffffu, b0 ? i2[0][j] : i2[1][j], 1);
        }
        const int row = tile0 + tg * RG_TG + ks;             // lane s finishes token s of the thread's eight
        if (row < row_end) {
#pragma unroll
            for (int j = 0; j < RG_OG; ++j) {
                const int o = o0 + oo + j;
                if (o >= bw) continue;
                const float r = rg_sigmoid(a1[j] + bra[j]), g = rg_sigmoid(i1[j] + bri[j]);
                const float log_a = -decay_scale * r * sp[j];
                const float keep = sqrtf(fmaxf(-expm1f(2.f * log_a), 0.f));
                const size_t at = (size_t)row * width + blk * bw + o;
                a_out[at] = expf(log_a);
                b_out[at] = keep * g * cur[o * us_ld + tg * RG_TG + ks];
            }
        }
        __syncthreads();                                     // this buffer is refilled by the next round's copies
    }
    rg_cp_async_wait_0();
}

// Blocks of channels too wide for the kernel above (their slices of weights and a tile of inputs pass shared
// memory): a tile of 8 tokens' inputs in shared memory, a thread per output channel, the weights read from global
// memory in input order.  Which of the two kernels runs follows from the block width alone, so a model's bits do not
// depend on the step.
#define RG_WIDE_TN 8
template <typename TW>
__global__ void __launch_bounds__(256)
rglru_gates_wide_kernel(const float* __restrict__ u, const TW* __restrict__ wa_t, const TW* __restrict__ wi_t,
                   const void* __restrict__ ba, const void* __restrict__ bi, const void* __restrict__ lam, int vec_dtype,
                   float decay_scale, float* __restrict__ a_out, float* __restrict__ b_out, int n_rows, int width,
                   int bw) {
    gi_pdl_start();
    extern __shared__ __align__(16) float us[];                  // [RG_WIDE_TN][bw]
    const int row0 = blockIdx.x * RG_WIDE_TN, blk = blockIdx.y;
    const int rows = min(RG_WIDE_TN, n_rows - row0);
    for (int i = threadIdx.x; i < RG_WIDE_TN * bw; i += blockDim.x) {
        const int t = i / bw, k = i - t * bw;
        us[i] = t < rows ? u[(size_t)(row0 + t) * width + blk * bw + k] : 0.f;
    }
    __syncthreads();
    const TW* wa = wa_t + (size_t)blk * bw * bw;
    const TW* wi = wi_t + (size_t)blk * bw * bw;
    for (int o = blockIdx.z * blockDim.x + threadIdx.x; o < bw; o += gridDim.z * blockDim.x) {
        float ra[RG_WIDE_TN], ri[RG_WIDE_TN];
#pragma unroll
        for (int t = 0; t < RG_WIDE_TN; ++t) ra[t] = ri[t] = 0.f;
        int k = 0;
        if (bw % 4 == 0) {
            for (; k < bw; k += 4) {
                float a4[4], i4[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    a4[j] = to_f32(wa[(size_t)(k + j) * bw + o]);
                    i4[j] = to_f32(wi[(size_t)(k + j) * bw + o]);
                }
#pragma unroll
                for (int t = 0; t < RG_WIDE_TN; ++t) {
                    const float4 x = *reinterpret_cast<const float4*>(us + t * bw + k);
                    ra[t] = fmaf(a4[0], x.x, ra[t]); ra[t] = fmaf(a4[1], x.y, ra[t]);
                    ra[t] = fmaf(a4[2], x.z, ra[t]); ra[t] = fmaf(a4[3], x.w, ra[t]);
                    ri[t] = fmaf(i4[0], x.x, ri[t]); ri[t] = fmaf(i4[1], x.y, ri[t]);
                    ri[t] = fmaf(i4[2], x.z, ri[t]); ri[t] = fmaf(i4[3], x.w, ri[t]);
                }
            }
        } else {
            for (; k < bw; ++k) {
                const float a1 = to_f32(wa[(size_t)k * bw + o]), i1 = to_f32(wi[(size_t)k * bw + o]);
#pragma unroll
                for (int t = 0; t < RG_WIDE_TN; ++t) {
                    ra[t] = fmaf(a1, us[t * bw + k], ra[t]);
                    ri[t] = fmaf(i1, us[t * bw + k], ri[t]);
                }
            }
        }
        const int c = blk * bw + o;
        const float bra = load_w(ba, vec_dtype, c), bri = load_w(bi, vec_dtype, c);
        const float sp = rg_softplus(load_w(lam, vec_dtype, c));
#pragma unroll
        for (int t = 0; t < RG_WIDE_TN; ++t) {
            if (t >= rows) break;
            const float r = rg_sigmoid(ra[t] + bra), g = rg_sigmoid(ri[t] + bri);
            const float log_a = -decay_scale * r * sp;
            const float a = expf(log_a);
            const float keep = sqrtf(fmaxf(-expm1f(2.f * log_a), 0.f));
            a_out[(size_t)(row0 + t) * width + c] = a;
            b_out[(size_t)(row0 + t) * width + c] = keep * g * us[t * bw + o];
        }
    }
}

// The same gates on tensor cores, for bfloat16 matrices.  A float32 input is the exact sum of three bfloat16 numbers
// (its 24 bits of mantissa cut into 8 + 8 + 8), every product of one of them with a bfloat16 weight is exact in float32,
// and three `mma.sync` sum 16 inputs' products from zero.  The sums of all inputs are made of those by adds that round to
// nearest: the tensor core cuts its sums off, and carried through all inputs that put b four to six times as far from 64
// bits as the kernels above with float32 multiply-adds.  Relative errors of b (2-norm) against 64 bits in units of 1e-8, those
// kernels / sums carried through / so, inputs of size 1: blocks of 64 7.6 / 10.8 / 7.5, 128 8.0 / 17.1 / 7.6, 320 8.8 / 38.9 / 8.0,
// 1,280 25 / 156 / 9.6; a's 3.2 / 3.2 to 5.4 / 3.2.
// A block of 8 warps takes 16 MW rows x 64 outputs of both gates; inputs and weights come through a ring of three chunks of
// 32 inputs.  Many rows: a warp has 16 rows and all 64 outputs, so that the split of its inputs serves 128 columns (MW 8).
// Few rows: the warps share the outputs of the same rows (MW 1: 8 outputs of both gates each), since one warp with all of
// them would have the products of a chunk to itself.  A row's sums are the same in every form and do not depend on the
// other rows, so its bits depend on the block width alone.
// Bound by the tensor pipe's legacy path and by the exponentials of the last step.  Measured in us, multiply-adds / always
// MW 8 / so: 16 blocks of 320, 2,494 rows 945 / 210 / 210, 64 rows 38 / 24 / 17, 8 rows 25 / 19 / 8; 64 blocks of 64, 8 rows
// 8.4 / 10.7 / 4.0, 64 rows 10.5 / 15 / 6.0; 16 blocks of 128, 64 rows 9.9 / 17 / 5.9, 512 rows 42 / 19 / 16.
#define RM_OUT 64
#define RM_KC 32
#define RM_STAGES 3
#define RM_ULD (RM_KC + 8)           // row length of the staged inputs: pairs of floats without bank conflicts
#define RM_WLD (RM_OUT + 8)          // of the staged weights: the rows that ldmatrix reads start 4 banks apart

// {x, y} as three pairs of bfloat16 that sum to them exactly: the upper 16 bits, the upper 16 bits of what is left, and the
// rest.  An infinity stays in the first (its remainder would be a NaN); a NaN's remainder is one, whatever its upper bits say.
__device__ __forceinline__ void rm_split(float2 v, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
    const uint32_t x = __float_as_uint(v.x), y = __float_as_uint(v.y);
    hi = __byte_perm(x, y, 0x7632);
    float rx = v.x - __uint_as_float(x & 0xffff0000u), ry = v.y - __uint_as_float(y & 0xffff0000u);
    if ((x & 0x7fffffffu) == 0x7f800000u) rx = 0.f;
    if ((y & 0x7fffffffu) == 0x7f800000u) ry = 0.f;
    const uint32_t mx = __float_as_uint(rx), my = __float_as_uint(ry);
    mid = __byte_perm(mx, my, 0x7632);
    lo = __byte_perm(__float_as_uint(rx - __uint_as_float(mx & 0xffff0000u)),
                     __float_as_uint(ry - __uint_as_float(my & 0xffff0000u)), 0x7632);
}
// d = a b + c
__device__ __forceinline__ void rm_mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1, const float (&c)[4]) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};"
                 : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(c[0]), "f"(c[1]), "f"(c[2]), "f"(c[3]));
}
// MW: warps along the rows, 16 rows each; the 8 / MW warps of the same rows share the 64 outputs, 8 MW each.
template <int MW>
__global__ void __launch_bounds__(256, 2)
rglru_gates_mma_kernel(const float* __restrict__ u, const bf16* __restrict__ wa_t, const bf16* __restrict__ wi_t,
                       const void* __restrict__ ba, const void* __restrict__ bi, const void* __restrict__ lam, int vec_dtype,
                       float decay_scale, float* __restrict__ a_out, float* __restrict__ b_out, int n_rows, int width, int bw) {
    constexpr int ROWS = 16 * MW, STAGE_BYTES = ROWS * RM_ULD * 4 + 2 * RM_KC * RM_WLD * 2;
    gi_pdl_start();
    extern __shared__ __align__(16) unsigned char rg_smem[];
    __shared__ float vecs[3][RM_OUT];                        // both biases and softplus(lam) of this block's outputs
    const int slices = (bw + RM_OUT - 1) / RM_OUT;           // neighbouring blocks share their rows' inputs
    const int o0 = (int)(blockIdx.x % slices) * RM_OUT, row0 = (int)(blockIdx.x / slices) * ROWS, blk = blockIdx.y;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int wr = warp % MW * 16, wc = warp / MW * (8 * MW);          // the warp's first row and output of the block
    const int chunks = (bw + RM_KC - 1) / RM_KC;
    auto stage_u = [&](int s) { return reinterpret_cast<float*>(rg_smem + (size_t)s * STAGE_BYTES); };
    auto stage_w = [&](int s) { return reinterpret_cast<bf16*>(rg_smem + (size_t)s * STAGE_BYTES + ROWS * RM_ULD * 4); };
    // A chunk's inputs and weights, 16 bytes at a time; what lies outside (rows, inputs or outputs beyond the last) is
    // zero-filled and its address is that of something inside.
    auto fetch = [&](int chunk) {
        if (chunk < chunks) {
            const int k0 = chunk * RM_KC, s = chunk % RM_STAGES;
            float* us = stage_u(s);
            bf16* ws = stage_w(s);
#pragma unroll
            for (int i = 0; i < (ROWS * (RM_KC / 4) + 255) / 256; ++i) {
                const int id = threadIdx.x + 256 * i, r = id / (RM_KC / 4), c = id % (RM_KC / 4) * 4;
                const bool in = row0 + r < n_rows && k0 + c < bw;
                if (r < ROWS) rg_cp_async_16(us + r * RM_ULD + c, u + (in ? (size_t)(row0 + r) * width + blk * bw + k0 + c : 0), in ? 16 : 0);
            }
#pragma unroll
            for (int i = 0; i < 2 * RM_KC * (RM_OUT / 8) / 256; ++i) {
                const int id = threadIdx.x + 256 * i, k = id / (RM_OUT / 8) % RM_KC, c = id % (RM_OUT / 8) * 8;
                const bf16* src = id >= RM_KC * (RM_OUT / 8) ? wi_t : wa_t;
                const bool in = k0 + k < bw && o0 + c < bw;
                rg_cp_async_16(ws + (id / (RM_OUT / 8)) * RM_WLD + c, src + (in ? ((size_t)blk * bw + k0 + k) * bw + o0 + c : 0), in ? 16 : 0);
            }
        }
        rg_cp_async_commit();                                // an empty group at the end: the count stays uniform
    };
    for (int c = 0; c < RM_STAGES - 1; ++c) fetch(c);
    if (threadIdx.x < RM_OUT) {
        const int c = blk * bw + min(o0 + (int)threadIdx.x, bw - 1);
        vecs[0][threadIdx.x] = load_w(ba, vec_dtype, c);
        vecs[1][threadIdx.x] = load_w(bi, vec_dtype, c);
        vecs[2][threadIdx.x] = rg_softplus(load_w(lam, vec_dtype, c));
    }
    float acc[2][MW][4];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < MW; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[i][j][e] = 0.f;
    const bool works = row0 + wr < n_rows && o0 + wc < bw;   // a warp whose rows or outputs lie beyond the last only copies
    const float zero[4] = {0.f, 0.f, 0.f, 0.f};
    for (int chunk = 0; chunk < chunks; ++chunk) {
        rg_cp_async_wait_1();
        __syncthreads();                                     // this chunk is there, and the one before it is done with
        fetch(chunk + RM_STAGES - 1);
        if (!works) continue;
        const float* us = stage_u(chunk % RM_STAGES) + (wr + g) * RM_ULD + 2 * t;
        const bf16* ws = stage_w(chunk % RM_STAGES) + wc;
#pragma unroll
        for (int kk = 0; kk < RM_KC; kk += 16) {
            uint32_t hi[4], mid[4], lo[4];
#pragma unroll
            for (int e = 0; e < 4; ++e)                      // rows g, g + 8; inputs 2 t, 2 t + 1 and 8 further
                rm_split(*reinterpret_cast<const float2*>(us + (e & 1) * 8 * RM_ULD + kk + (e >> 1) * 8), hi[e], mid[e], lo[e]);
            auto products = [&](float (&sum)[4], uint32_t b0, uint32_t b1) {
                float d[4];
                rm_mma(d, lo, b0, b1, zero);
                rm_mma(d, mid, b0, b1, d);
                rm_mma(d, hi, b0, b1, d);
#pragma unroll
                for (int e = 0; e < 4; ++e) sum[e] += d[e];
            };
#pragma unroll
            for (int gate = 0; gate < 2; ++gate)
                if (MW == 1) {
                    uint32_t b[2];
                    const bf16* at = ws + (gate * RM_KC + kk + (lane & 15)) * RM_WLD;
                    asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];"
                                 : "=r"(b[0]), "=r"(b[1]) : "r"((uint32_t)__cvta_generic_to_shared(at)));
                    products(acc[gate][0], b[0], b[1]);
                } else {
#pragma unroll
                    for (int j = 0; j + 1 < MW; j += 2) {
                        uint32_t b[4];
                        const bf16* at = ws + (gate * RM_KC + kk + (lane & 15)) * RM_WLD + j * 8 + (lane >> 4) * 8;
                        asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                                     : "=r"(b[0]), "=r"(b[1]), "=r"(b[2]), "=r"(b[3]) : "r"((uint32_t)__cvta_generic_to_shared(at)));
                        products(acc[gate][j], b[0], b[1]);
                        products(acc[gate][j + 1], b[2], b[3]);
                    }
                }
        }
    }
    rg_cp_async_wait_0();
    if (!works) return;
#pragma unroll
    for (int j = 0; j < MW; ++j) {
        const int oo = wc + j * 8 + 2 * t, o = o0 + oo;
        if (o >= bw) continue;                               // a multiple of 8: the pair's other output is in as well
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const int row = row0 + wr + g + half * 8;
            if (row >= n_rows) continue;
            const size_t at = (size_t)row * width + blk * bw + o;
            const float2 x = *reinterpret_cast<const float2*>(u + at);
            float2 ra, rb;
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                float za = acc[0][j][half * 2 + e], zi = acc[1][j][half * 2 + e];
                if (za != za || zi != zi) {
                    za = rm_plain(u + at - o, wa_t + (size_t)blk * bw * bw + o + e, bw);
                    zi = rm_plain(u + at - o, wi_t + (size_t)blk * bw * bw + o + e, bw);
                }
                const float r = rg_sigmoid(za + vecs[0][oo + e]), i = rg_sigmoid(zi + vecs[1][oo + e]);
                const float log_a = -decay_scale * r * vecs[2][oo + e];
                const float keep = sqrtf(fmaxf(-expm1f(2.f * log_a), 0.f));
                (e ? ra.y : ra.x) = expf(log_a);
                (e ? rb.y : rb.x) = keep * i * (e ? x.y : x.x);
            }
            *reinterpret_cast<float2*>(a_out + at) = ra;
            *reinterpret_cast<float2*>(b_out + at) = rb;
        }
    }
}

extern "C" int gi_rglru_gates(const float* u, const void* wa_t, const void* wi_t, int w_dtype, const void* ba,
                              const void* bi, const void* lam, int vec_dtype, float decay_scale, float* a_out,
                              float* b_out, int n_rows, int width, int blocks, void* stream) {
    GI_REQUIRE(n_rows >= 0 && width > 0 && blocks > 0 && width % blocks == 0, "gi_rglru_gates: %d channels in %d blocks", width, blocks);
    GI_REQUIRE(blocks <= 65535, "gi_rglru_gates: %d blocks is beyond 65535", blocks);
    GI_REQUIRE(w_dtype == GI_DTYPE_F32 || w_dtype == GI_DTYPE_BF16, "gi_rglru_gates: weight dtype %d", w_dtype);
    if (n_rows == 0) return 0;
    const int bw = width / blocks;
    const size_t wsize = w_dtype == GI_DTYPE_F32 ? 4 : 2;
    // bfloat16 matrices whose rows are whole 16-byte words: tensor cores.  (float32 matrices would need three parts as
    // well, and nine products.)
    if (w_dtype == GI_DTYPE_BF16 && bw % 8 == 0 && ((uintptr_t)u | (uintptr_t)wa_t | (uintptr_t)wi_t) % 16 == 0 &&
        ((uintptr_t)a_out | (uintptr_t)b_out) % 8 == 0) {
        // the tallest tile that rows fill by more than a half and that leaves an SM each a block of threads
        const long long across = (long long)((bw + RM_OUT - 1) / RM_OUT) * blocks;
        int mw = 8;
        while (mw > 1 && (n_rows <= 8 * mw || across * ((n_rows + 16 * mw - 1) / (16 * mw)) < 148)) mw /= 2;
#define RM_LAUNCH(MW) do {                                                                                                     \
            const size_t smem = (size_t)RM_STAGES * (16 * MW * RM_ULD * 4 + 2 * RM_KC * RM_WLD * 2);                           \
            if (int rc = gi_reserve_smem((const void*)rglru_gates_mma_kernel<MW>, smem, "gi_rglru_gates")) return rc;          \
            dim3 grid((unsigned)((bw + RM_OUT - 1) / RM_OUT) * (unsigned)((n_rows + 16 * MW - 1) / (16 * MW)), blocks);        \
            gi_launch(rglru_gates_mma_kernel<MW>, grid, dim3(256), smem, (cudaStream_t)stream, u, (const bf16*)wa_t,           \
                      (const bf16*)wi_t, ba, bi, lam, vec_dtype, decay_scale, a_out, b_out, n_rows, width, bw);                \
        } while (0)
        if (mw == 1) RM_LAUNCH(1);
        else if (mw == 2) RM_LAUNCH(2);
        else if (mw == 4) RM_LAUNCH(4);
        else RM_LAUNCH(8);
#undef RM_LAUNCH
        return gi_check_launch("gi_rglru_gates");
    }
    // outputs per block of threads and tokens per tile: as many as shared memory takes (the sizes depend on the
    // block width alone, never on the step)
    int orange = 32, tt = 32;
    auto smem_of = [&](int orng, int t) {
        return (((size_t)2 * bw * (orng + RG_WPAD) * wsize + 15) & ~(size_t)15) + (size_t)2 * bw * (t + 4) * sizeof(float);
    };
    while (smem_of(orange, tt) > 200 * 1024 && tt > 16) tt /= 2;
    while (smem_of(orange, tt) > 200 * 1024 && orange > 16) orange /= 2;      // beyond that: the kernel for wide blocks
    cudaStream_t s = (cudaStream_t)stream;
    if (smem_of(orange, tt) > 200 * 1024) {
        const size_t smem = (size_t)RG_WIDE_TN * bw * sizeof(float);
        GI_REQUIRE(smem <= 200 * 1024, "gi_rglru_gates: blocks of %d channels do not fit shared memory", bw);
        const int threads = bw >= 256 ? 256 : (bw + 31) / 32 * 32;
        const int tiles = (n_rows + RG_WIDE_TN - 1) / RG_WIDE_TN;
        int cut = 1;
        while (cut * threads < bw && (long long)tiles * blocks * cut < 296) ++cut;
        dim3 grid(tiles, blocks, cut);
        if (w_dtype == GI_DTYPE_F32) {
            if (int rc = gi_reserve_smem((const void*)rglru_gates_wide_kernel<float>, smem, "gi_rglru_gates")) return rc;
            gi_launch(rglru_gates_wide_kernel<float>, grid, dim3(threads), smem, s, u, (const float*)wa_t, (const float*)wi_t,
                      ba, bi, lam, vec_dtype, decay_scale, a_out, b_out, n_rows, width, bw);
        } else {
            if (int rc = gi_reserve_smem((const void*)rglru_gates_wide_kernel<bf16>, smem, "gi_rglru_gates")) return rc;
            gi_launch(rglru_gates_wide_kernel<bf16>, grid, dim3(threads), smem, s, u, (const bf16*)wa_t, (const bf16*)wi_t,
                      ba, bi, lam, vec_dtype, decay_scale, a_out, b_out, n_rows, width, bw);
        }
        return gi_check_launch("gi_rglru_gates");
    }
    const int threads = RG_KS * (orange / RG_OG) * (tt / RG_TG);
    const int slices = (bw + orange - 1) / orange;
    // many rows: the rows are cut over the grid's third axis until there are about eight blocks of threads to an SM
    // one after the other (an SM holds one or two at a time; with fewer, longer ones the last round would leave most
    // SMs idle, and a block's own copy of its weights costs little)
    const int tiles = (n_rows + tt - 1) / tt;
    long long cut = (8LL * 148 + (long long)blocks * slices - 1) / ((long long)blocks * slices);
    cut = cut < 1 ? 1 : (cut > tiles ? tiles : (cut > 65535 ? 65535 : cut));
    const int rows_per_cta = (int)((tiles + cut - 1) / cut) * tt;
    dim3 grid(blocks, slices, (unsigned)((n_rows + rows_per_cta - 1) / rows_per_cta));
    const size_t smem = smem_of(orange, tt);
    if (w_dtype == GI_DTYPE_F32) {
        if (int rc = gi_reserve_smem((const void*)rglru_gates_kernel<float>, smem, "gi_rglru_gates")) return rc;
        gi_launch(rglru_gates_kernel<float>, grid, dim3(threads), smem, s, u, (const float*)wa_t, (const float*)wi_t, ba, bi,
                  lam, vec_dtype, decay_scale, a_out, b_out, n_rows, width, bw, orange, tt, rows_per_cta);
    } else {
        if (int rc = gi_reserve_smem((const void*)rglru_gates_kernel<bf16>, smem, "gi_rglru_gates")) return rc;
        gi_launch(rglru_gates_kernel<bf16>, grid, dim3(threads), smem, s, u, (const bf16*)wa_t, (const bf16*)wi_t, ba, bi,
                  lam, vec_dtype, decay_scale, a_out, b_out, n_rows, width, bw, orange, tt, rows_per_cta);
    }
    return gi_check_launch("gi_rglru_gates");
}

// The gate branch's activation, the tanh form of gelu: with the library's tanh for a float32 engine; for bfloat16
// (the activation of a projection, whose result is rounded to 8 bits of mantissa right after) with the hardware's
// approximate tanh, which is good to about 11 bits.
template <typename T> __device__ __forceinline__ float rg_gate_act(float z) { return rg_gelu_tanh(z); }
template <> __device__ __forceinline__ float rg_gate_act<bf16>(float z) {
    float t;
    asm("tanh.approx.f32 %0, %1;" : "=f"(t) : "f"(0.7978845608028654f * (z + 0.044715f * z * z * z)));
    return 0.5f * z * (1.f + t);
}

// spans [n_seq, 3] = {slot, first row, rows}, or null: every row is a sequence of its own with the slot of tok_slot.
//
// A block of one warp walks 32 channels of a sequence (one long prompt of a few thousand channels then reaches every SM);
// the inputs of the next 60 tokens are under way into shared memory by asynchronous copies, in groups of four tokens (three
// copies of 16 bytes a lane).  What bounds a walk is a trip to memory divided by the tokens under way.  Loads into
// registers could not keep 32 tokens under way however they were written: a warp has six counters for loads under way, and
// waiting for one group's waits for every later load on the same counter.  Measured with 2,494 rows of 5,120 channels in four
// prompts of up to 900 tokens (153 MB): 144 us with the ring in registers, 63 us so.  Rows that do not start on 16 bytes
// are copied 4 bytes a lane (a, b and y each by its own alignment): 129 us with y in columns from the fourth on, 83 us in
// float32 from the first; loads that a group waited for took 205 and 221 us.
#define RG_SUB 4             // tokens to a group
#define RG_DEPTH 16          // groups in the ring
#define RG_SCAN_THREADS 32
#define RG_YLD 40            // row length of the staged y: 32 elements, one more where a row starts inside a word, rows on 16 bytes
template <typename T>
__global__ void __launch_bounds__(RG_SCAN_THREADS)
rglru_scan_kernel(const float* __restrict__ a, const float* __restrict__ b, const T* __restrict__ y, long long ldy,
                  const void* __restrict__ y_bias, int bias_dtype, float* __restrict__ state, long long state_stride,
                  const int* __restrict__ spans, const int* __restrict__ tok_slot, T* __restrict__ out, long long ldo,
                  int width, int wide) {
    gi_pdl_start();
    const int lane = threadIdx.x, cw = blockIdx.y * RG_SCAN_THREADS, c = cw + lane;
    const bool live = c < width;
    int slot, start, len;
    if (spans) { slot = spans[3 * blockIdx.x]; start = spans[3 * blockIdx.x + 1]; len = spans[3 * blockIdx.x + 2]; }
    else { slot = tok_slot[blockIdx.x]; start = blockIdx.x; len = 1; }
    if (slot < 0) {
        for (int t = 0; t < len && live; ++t) out[(size_t)(start + t) * ldo + c] = from_f32<T>(0.f);
        return;
    }
    const float yb = y_bias && live ? load_w(y_bias, bias_dtype, c) : 0.f;
    float S = live ? state[(size_t)slot * state_stride + c] : 0.f;
    if (len == 1) {                                          // a decode step's row: nothing to run ahead of
        if (!live) return;
        const size_t r = (size_t)start;
        S = fmaf(a[r * width + c], S, b[r * width + c]);
        out[r * ldo + c] = from_f32<T>(S * rg_gate_act<T>(to_f32(y[r * ldy + c]) + yb));
        state[(size_t)slot * state_stride + c] = S;
        return;
    }
    __shared__ __align__(16) float a_s[RG_DEPTH][RG_SUB][32], b_s[RG_DEPTH][RG_SUB][32];
    __shared__ __align__(16) T y_s[RG_DEPTH][RG_SUB][RG_YLD];
    const int groups = (len + RG_SUB - 1) / RG_SUB;
    // 1 for a row of bfloat16 y that starts in the middle of a 4-byte word: its elements lie one place further in y_s
    auto y_row = [&](int t) { return y + (size_t)(start + min(t, len - 1)) * ldy + cw; };
    auto y_shift = [&](const T* row) { return sizeof(T) == 2 ? (int)((uintptr_t)row >> 1 & 1) : 0; };
    // lane l copies 16 bytes of token l / 8 of a group (bytes beyond the last channel are zero-filled); a group's last
    // tokens beyond the sequence are its last row again, and not walked
    auto fetch = [&](int grp) {
        if (grp < groups) {
            const int s = grp % RG_DEPTH;
            if (wide & 1) {
                const int j = lane >> 3, o = (lane & 7) * 4, n = min(16, max(0, (width - cw - o) * 4));
                const size_t at = (size_t)(start + min(grp * RG_SUB + j, len - 1)) * width + (n ? cw + o : 0);
                rg_cp_async_16(&a_s[s][j][o], a + at, n);
                rg_cp_async_16(&b_s[s][j][o], b + at, n);
            } else {
#pragma unroll
                for (int j = 0; j < RG_SUB; ++j) {           // rows that do not start on 16 bytes: a float a lane
                    const size_t at = (size_t)(start + min(grp * RG_SUB + j, len - 1)) * width + (live ? c : 0);
                    rg_cp_async_4n(&a_s[s][j][lane], a + at, live ? 4 : 0);
                    rg_cp_async_4n(&b_s[s][j][lane], b + at, live ? 4 : 0);
                }
            }
            if (wide & 2) {
                constexpr int PER = 16 / (int)sizeof(T), LPR = 32 / PER;       // elements to a copy, lanes to a row
                if (lane < RG_SUB * LPR) {
                    const int jy = lane / LPR, oy = lane % LPR * PER, ny = min(16, max(0, (width - cw - oy) * (int)sizeof(T)));
                    rg_cp_async_16(&y_s[s][jy][oy], y_row(grp * RG_SUB + jy) + (ny ? oy : -cw), ny);
                }
            } else {
                // A row's elements by whole 4-byte words of memory, a word a lane: the first may hold the element in front of
                // the row (a part of the same aligned word, so of the same allocation), the last is cut off at the row's end.
                constexpr int PER = 4 / (int)sizeof(T), WORDS = 32 / PER + (PER > 1);
#pragma unroll
                for (int j = 0; j < RG_SUB; ++j) {
                    const T* row = y_row(grp * RG_SUB + j);
                    const int sh = y_shift(row), ny = min(4, max(0, (min(32, width - cw) + sh - lane * PER) * (int)sizeof(T)));
                    if (lane < WORDS) rg_cp_async_4n(&y_s[s][j][lane * PER], row - sh + (ny ? lane * PER : 0), ny);
                }
            }
        }
        rg_cp_async_commit();
    };
    for (int g = 0; g < RG_DEPTH - 1; ++g) fetch(g);
    T* dst = out + (size_t)start * ldo + c;
    for (int grp = 0; grp < groups; ++grp) {
        asm volatile("cp.async.wait_group %0;\n" ::"n"(RG_DEPTH - 2));
        __syncwarp();                                        // every lane's copies of this group, and the last group's reads
        fetch(grp + RG_DEPTH - 1);
        // The chain of dependent multiply-adds alone, then what waits for nothing, all four tokens of it side by side and
        // outside any branch: a warp has its scheduler nearly to itself, so a serial step costs its whole latency.
        const int s = grp % RG_DEPTH, left = len - grp * RG_SUB;
        float ga[RG_SUB], gb[RG_SUB], gy[RG_SUB];
#pragma unroll
        for (int j = 0; j < RG_SUB; ++j) {
            ga[j] = a_s[s][j][lane];
            gb[j] = b_s[s][j][lane];
            gy[j] = rg_gate_act<T>(to_f32(y_s[s][j][lane + (wide & 2 ? 0 : y_shift(y_row(grp * RG_SUB + j)))]) + yb);
        }
#pragma unroll
        for (int j = 0; j < RG_SUB; ++j) {
            S = fmaf(j < left ? ga[j] : 1.f, S, j < left ? gb[j] : 0.f);      // beyond the sequence: S stays as it is
            gy[j] *= S;
        }
        T v[RG_SUB];
#pragma unroll
        for (int j = 0; j < RG_SUB; ++j) v[j] = from_f32<T>(gy[j]);
#pragma unroll
        for (int j = 0; j < RG_SUB; ++j)
            if (j < left && live) dst[(size_t)j * ldo] = v[j];
        dst += (size_t)RG_SUB * ldo;
    }
    rg_cp_async_wait_0();
    if (live) state[(size_t)slot * state_stride + c] = S;
}

extern "C" int gi_rglru_scan(const float* a, const float* b, const void* y, long long ldy, int act_dtype, const void* y_bias,
                             int bias_dtype, float* state, long long state_stride, const int* spans, const int* tok_slot,
                             void* out, long long ldo, int n_seqs, int width, void* stream) {
    GI_REQUIRE(n_seqs >= 0 && width > 0 && ldy >= width && ldo >= width && state_stride >= width, "gi_rglru_scan: sizes");
    GI_REQUIRE((width + RG_SCAN_THREADS - 1) / RG_SCAN_THREADS <= 65535, "gi_rglru_scan: %d channels", width);
    if (n_seqs == 0) return 0;
    dim3 grid(n_seqs, (width + RG_SCAN_THREADS - 1) / RG_SCAN_THREADS);
    const int item = act_dtype == GI_DTYPE_F32 ? 4 : 2;
    // 1: rows of a and b start on 16 bytes, 2: rows of y do
    const int wide = (width % 4 == 0 && ((uintptr_t)a | (uintptr_t)b) % 16 == 0 ? 1 : 0) | (ldy * item % 16 == 0 && (uintptr_t)y % 16 == 0 ? 2 : 0);
    cudaStream_t s = (cudaStream_t)stream;
    if (act_dtype == GI_DTYPE_F32)
        gi_launch(rglru_scan_kernel<float>, grid, dim3(RG_SCAN_THREADS), 0, s, a, b, (const float*)y, ldy, y_bias, bias_dtype, state,
                  state_stride, spans, tok_slot, (float*)out, ldo, width, wide);
    else if (act_dtype == GI_DTYPE_BF16)
        gi_launch(rglru_scan_kernel<bf16>, grid, dim3(RG_SCAN_THREADS), 0, s, a, b, (const bf16*)y, ldy, y_bias, bias_dtype, state,
                  state_stride, spans, tok_slot, (bf16*)out, ldo, width, wide);
    else
        GI_REQUIRE(false, "gi_rglru_scan: activation dtype %d", act_dtype);
    return gi_check_launch("gi_rglru_scan");
}
