// The gated delta rule over prompts, 16 tokens at a time (recurrent.cu has the recurrence token by token, which decode steps, short
// portions and the 32-bit engine run).
//
// With G_t the product of a chunk's decays up to token t, channel by channel, and S the state in front of the chunk (rows are value
// columns), the chunk's updates u_t and outputs o_t are
//   A[t][s] = sum over channels of k_t k_s (decays s+1 .. t),  B[t][s] likewise with q_t (s <= t)
//   u = T V - (T KG) S,   T = (1 + beta A)^-1 beta by forward substitution, KG_t = k_t G_t
//   o = QG S + B u,       QG_t = q_t G_t
//   S <- G_16 S + sum over s of u_s KE_s,  KE_s = k_s (decays s+1 .. 16)
// Products of decays are made as products or as exponentials of sums (never as quotients), so that none is beyond 1 and a decay of zero
// is exact.
// delta_chunk_prepare_kernel makes everything that does not depend on S, for all chunks and heads at once; delta_chunk_walk_kernel
// goes from chunk to chunk with S in registers.
//
// The products with S and u keep float32: every factor is cut into three bfloat16 parts that sum to it exactly (t5_split3 says where not),
// the six largest products run on `mma.sync` from zero, small ones first (the error of a product is below 2^-25), and what they give
// meets S by float32 multiply-adds.  The operands lie in memory as the tensor core's fragments, so that a lane reads its own 16 bytes.
// Measured, 2,048 tokens, 16 heads of 128 x 128, a decay per channel: 382 us token by token (a chain of 174 ns a token), 188 us so (the
// preparation 71, the walk 121).  Relative error (2-norm) of outputs / states against 64 bits in units of 1e-7, 600 tokens, token by token and
// so, by what softplus is taken of: around -9 (decays near 1, a memory of thousands of tokens) 22 / 29 and 2.1 / 2.2, -4 2.3 / 2.1 and 1.6 / 1.2,
// -2 1.50 / 1.21 and 1.45 / 1.02, 0 (a state is halved by a token) 1.25 / 0.85 and 1.30 / 0.88, 3 1.19 / 0.72 and 1.19 / 0.71.  With decays as products of
// rounded decays, what a token takes off straight from its value, and a token's own part among the tensor core's sums it was 170 us and
// 20 / 26, 2.2 / 2.0, 1.65 / 1.34, 1.52 / 1.08, 1.38 / 0.96.
#include "scan.cuh"
#include "tcgen05.cuh"

#define DC_T 16                      // tokens to a chunk
#define DC_STAGES 4                  // three at least: a chunk's copies are waited for while the one before is walked
#define DC_COLS 16                   // value columns to a block of the walk
#define DC_LD 136                    // floats of a row in the preparation's shared memory: 8 banks from row to row
#define DC_ERR_WAIT 81

// bytes of a chunk of one head: fragments of [T KG; QG] (32 rows), of KE without its last token's row, of B without its diagonal, G_16, the
// last token's key and B's diagonal as floats; then T V in slices of 16 columns.  (What a token has of itself, in an output and in
// the state behind it, joins the other sums last by a float32 multiply-add: where little is left of the state it is all but the result,
// and the tensor core, which cuts its sums off, would cut it.)
template <int D> struct DcChunk {
    static constexpr int FA = 32 * D * 6, FU = DC_T * D * 6, FB = DC_T * DC_T * 6, G = D * 4, KL = D * 4, BD = DC_T * 4;
    static constexpr int AT_G = FA + FU + FB, AT_KL = AT_G + G, AT_BD = AT_KL + KL, HEAD = AT_BD + BD;
};

// rows of sequence i in this launch's window, and its first chunk
struct DcSpan { int slot, start, len, chunk0; };
__device__ __forceinline__ int dc_chunks(const int* spans, int i, int row0, int row1) {
    const int a = max(spans[3 * i + 1], row0), b = min(spans[3 * i + 1] + spans[3 * i + 2], row1);
    return max(0, b - a + DC_T - 1) / DC_T;
}
__device__ __forceinline__ DcSpan dc_span(const int* __restrict__ spans, int i, int row0, int row1) {
    DcSpan s = {spans[3 * i], max(spans[3 * i + 1], row0), 0, 0};
    s.len = min(spans[3 * i + 1] + spans[3 * i + 2], row1) - s.start;
    for (int j = 0; j < i; ++j) s.chunk0 += dc_chunks(spans, j, row0, row1);
    return s;
}

template <int D, int CH>
__global__ void __launch_bounds__(128, 4)
delta_chunk_prepare_kernel(const float* __restrict__ qkv, long long ldq, int q_off, int k_off, int v_off, const float* __restrict__ ab,
                           long long ldab, int b_off, int a_off, const float* __restrict__ al, long long ldal,
                           const void* __restrict__ A_log, const void* __restrict__ dt_bias, int p_dtype, const int* __restrict__ spans, int n_seq,
                           unsigned char* __restrict__ chunks, int H, int Hk, int dv, float unit_eps, float q_scale, int row0, int row1) {
    gi_pdl_start();
    extern __shared__ __align__(16) float dc_smem[];
    float *q_s = dc_smem, *k_s = q_s + DC_T * DC_LD, *g_s = k_s + DC_T * DC_LD, *kg_s = g_s + DC_T * DC_LD, *ke_s = kg_s + DC_T * DC_LD;
    __shared__ __align__(16) float A_s[DC_T][DC_T], B_s[DC_T][DC_T];
    __shared__ float beta_s[DC_T], diag_s[DC_T];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, h = blockIdx.y, kh = h / (H / Hk);
    // which sequence this chunk is of
    int seq = 0, c = blockIdx.x;
    for (; seq < n_seq; ++seq) {
        const int n = dc_chunks(spans, seq, row0, row1);
        if (c < n) break;
        c -= n;
    }
    if (seq == n_seq || spans[3 * seq] < 0) return;
    const int first = max(spans[3 * seq + 1], row0) + c * DC_T, len = min(DC_T, min(spans[3 * seq + 1] + spans[3 * seq + 2], row1) - first);

    // everything is asked for first: a warp's four tokens of q, k and the decays' logits, a thread's value column
    constexpr int TW = DC_T / 4;
    const int ch = lane * 4, chd = min(ch, D - 4);
    float4 q4[TW], k4[TW], a4[TW];
    float b1[TW], v1[DC_T];
#pragma unroll
    for (int i = 0; i < TW; ++i) {
        const size_t r = first + min(warp * TW + i, len - 1);
        q4[i] = *reinterpret_cast<const float4*>(qkv + r * ldq + q_off + kh * D + chd);
        k4[i] = *reinterpret_cast<const float4*>(qkv + r * ldq + k_off + kh * D + chd);
        const float* a = al + r * ldal + a_off + (CH ? h * D + chd : h);
        if (CH) a4[i] = make_float4(a[0], a[1], a[2], a[3]);
        else a4[i] = make_float4(a[0], 0.f, 0.f, 0.f);
        b1[i] = ab[r * ldab + b_off + h];
    }
    auto values = [&](int col) {
#pragma unroll
        for (int t = 0; t < DC_T; ++t) v1[t] = qkv[(size_t)(first + min(t, len - 1)) * ldq + v_off + h * dv + col];
    };
    values(min(tid, dv - 1));
    float4 d4;
    if (CH) d4 = make_float4(load_w(dt_bias, p_dtype, h * D + chd), load_w(dt_bias, p_dtype, h * D + chd + 1),
                             load_w(dt_bias, p_dtype, h * D + chd + 2), load_w(dt_bias, p_dtype, h * D + chd + 3));
    else d4.x = load_w(dt_bias, p_dtype, h);
    const float rate = expf(load_w(A_log, p_dtype, h));
    // q and k as unit vectors, decays, beta.  A token beyond the sequence's end changes nothing.
#pragma unroll
    for (int i = 0; i < TW; ++i) {
        const int t = warp * TW + i;
        const bool in = t < len;
        float4 q = make_float4(0.f, 0.f, 0.f, 0.f), k = q, g = make_float4(1.f, 1.f, 1.f, 1.f);
        if (in && ch < D) { q = q4[i]; k = k4[i]; }
        float4 log_g = make_float4(0.f, 0.f, 0.f, 0.f);
        if (in) {
            log_g.x = -rate * rc_softplus(a4[i].x + d4.x);
            g.x = expf(log_g.x);
            if (CH) {
                log_g.y = -rate * rc_softplus(a4[i].y + d4.y);
                log_g.z = -rate * rc_softplus(a4[i].z + d4.z);
                log_g.w = -rate * rc_softplus(a4[i].w + d4.w);
                g.y = expf(log_g.y);
                g.z = expf(log_g.z);
                g.w = expf(log_g.w);
            } else {
                log_g.y = log_g.z = log_g.w = log_g.x;
                g.y = g.z = g.w = g.x;
            }
        }
        float sq = 0.f, sk = 0.f;
        sq = fmaf(q.x, q.x, sq); sq = fmaf(q.y, q.y, sq); sq = fmaf(q.z, q.z, sq); sq = fmaf(q.w, q.w, sq);
        sk = fmaf(k.x, k.x, sk); sk = fmaf(k.y, k.y, sk); sk = fmaf(k.z, k.z, sk); sk = fmaf(k.w, k.w, sk);
        sq = warp_sum(sq);
        sk = warp_sum(sk);
        // (a token beyond the end is zeros also where unit_eps is zero)
        const float iq = in ? q_scale / sqrtf(sq + unit_eps) : 0.f, ik = in ? 1.f / sqrtf(sk + unit_eps) : 0.f;
        if (ch < D) {
            *reinterpret_cast<float4*>(q_s + t * DC_LD + ch) = make_float4(q.x * iq, q.y * iq, q.z * iq, q.w * iq);
            *reinterpret_cast<float4*>(k_s + t * DC_LD + ch) = make_float4(k.x * ik, k.y * ik, k.z * ik, k.w * ik);
            *reinterpret_cast<float4*>(g_s + t * DC_LD + ch) = g;
            *reinterpret_cast<float4*>(kg_s + t * DC_LD + ch) = log_g;
        }
        if (lane == 0) beta_s[t] = in ? rc_sigmoid(b1[i]) : 0.f;
    }
    __syncthreads();

    // A and B: 8 lanes to a key s; its key, decayed token by token, against the keys and queries behind it
    {
        const int s = tid >> 3, part = tid & 7;
        constexpr int P = 8, N4 = D / 32;                    // words of four to a lane
        t5_f2 w[2 * N4];
        auto words = [&](const float* row, int i, t5_f2& x, t5_f2& y) {
            const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(row + KEY_OF(i, part));
            x = v.x;
            y = v.y;
        };
#pragma unroll
        for (int i = 0; i < N4; ++i) words(k_s + s * DC_LD, i, w[2 * i], w[2 * i + 1]);
        float ka[DC_T], qa[DC_T];
#pragma unroll
        for (int t = 0; t < DC_T; ++t) {
            ka[t] = qa[t] = 0.f;
            if (t < warp * 4) continue;                      // in front of this warp's first key
            t5_f2 k2[2] = {0ull, 0ull}, q2[2] = {0ull, 0ull}, x, y;
#pragma unroll
            for (int i = 0; i < N4; ++i) {
                words(g_s + t * DC_LD, i, x, y);
                if (t > s) {
                    w[2 * i] = t5_mul2(w[2 * i], x);
                    w[2 * i + 1] = t5_mul2(w[2 * i + 1], y);
                }
                words(k_s + t * DC_LD, i, x, y);
                k2[0] = t5_fma2(x, w[2 * i], k2[0]);
                k2[1] = t5_fma2(y, w[2 * i + 1], k2[1]);
                words(q_s + t * DC_LD, i, x, y);
                q2[0] = t5_fma2(x, w[2 * i], q2[0]);
                q2[1] = t5_fma2(y, w[2 * i + 1], q2[1]);
            }
            float lo, hi;
            t5_apart(t5_add2(k2[0], k2[1]), lo, hi);
            ka[t] = lo + hi;
            t5_apart(t5_add2(q2[0], q2[1]), lo, hi);
            qa[t] = lo + hi;
        }
#pragma unroll
        for (int half = 0; half < 2; ++half) {               // token `part` of eight ends in lane `part`
            const int t = half * 8 + part;
            const float a = part_sum_tokens<P>(*reinterpret_cast<float (*)[P]>(ka + half * 8), part);
            const float b = part_sum_tokens<P>(*reinterpret_cast<float (*)[P]>(qa + half * 8), part);
            A_s[t][s] = t > s ? a : 0.f;
            B_s[t][s] = t > s ? b : 0.f;
            if (t == s) diag_s[t] = b;
        }
    }
    __syncthreads();

    // x <- (1 + beta A)^-1 beta x by forward substitution.  What is taken off a number is summed up first: keys are unit vectors, so it is
    // a fraction of the number, and so are its roundings.
    auto substitute = [&](float (&x)[DC_T]) {
#pragma unroll
        for (int t = 0; t < DC_T; ++t) {
            float off = 0.f;
#pragma unroll
            for (int s = 0; s < t; s += 4) {
                const float4 a = *reinterpret_cast<const float4*>(&A_s[t][s]);       // zero from t on
                off = fmaf(a.x, x[s], off);
                if (s + 1 < t) off = fmaf(a.y, x[s + 1], off);
                if (s + 2 < t) off = fmaf(a.z, x[s + 2], off);
                if (s + 3 < t) off = fmaf(a.w, x[s + 3], off);
            }
            x[t] = (x[t] - off) * beta_s[t];
        }
    };
    // T V: a thread takes a value column; a lane of the walk finds its eight tokens and columns side by side
    unsigned char* chunk = chunks + ((size_t)blockIdx.x * H + h) * (size_t)(DcChunk<D>::HEAD + DC_T * 4 * dv);
    float4* tv = reinterpret_cast<float4*>(chunk + DcChunk<D>::HEAD);
    for (int col0 = 0; col0 < dv; col0 += 128) {
        const int col = col0 + tid;
        if (col0) values(min(col, dv - 1));
#pragma unroll
        for (int t = 0; t < DC_T; ++t) v1[t] = t < len ? v1[t] : 0.f;
        substitute(v1);
        if (col0) __syncthreads();
        float* dst = ke_s + (tid >> 4) * 256 + (tid & 7) * 32 + (tid >> 3 & 1) * 4;
#pragma unroll
        for (int i = 0; i < 4; ++i)                          // tokens 2 i, 2 i + 1, and those 8 later
            *reinterpret_cast<float4*>(dst + i * 8) = make_float4(v1[2 * i], v1[2 * i + 1], v1[2 * i + 8], v1[2 * i + 9]);
        __syncthreads();
        for (int i = tid; i < min(dv - col0, 128) * DC_T / 4; i += 128) tv[col0 * DC_T / 4 + i] = reinterpret_cast<const float4*>(ke_s)[i];
    }
    __syncthreads();
    // a thread takes a channel: its products of decays as exponentials of sums (a product of decays near 1 would keep the rounding of
    // every one of them, the same way for all tokens of a long memory), and T KG
    if (tid < D) {
        float l[DC_T], x[DC_T], sum = 0.f, run = 1.f;
#pragma unroll
        for (int t = 0; t < DC_T; ++t) {
            l[t] = kg_s[t * DC_LD + tid];
            sum += l[t];
            run = expf(sum);
            x[t] = k_s[t * DC_LD + tid] * run;
            q_s[t * DC_LD + tid] *= run;
        }
        reinterpret_cast<float*>(chunk + DcChunk<D>::AT_G)[tid] = run;
        reinterpret_cast<float*>(chunk + DcChunk<D>::AT_KL)[tid] = k_s[(len - 1) * DC_LD + tid];
        sum = 0.f;
#pragma unroll
        for (int t = DC_T - 1; t >= 0; --t) {
            ke_s[t * DC_LD + tid] = t == len - 1 ? 0.f : k_s[t * DC_LD + tid] * expf(sum);
            sum += l[t];
        }
        substitute(x);
#pragma unroll
        for (int t = 0; t < DC_T; ++t) kg_s[t * DC_LD + tid] = x[t];
    }
    __syncthreads();

    // fragments.  Of the 32 rows [T KG; QG]: item (group of channels, 16 of its channels, two tiles of 8 rows, lane)
    constexpr int KS = D / 64;
    uint4* fa = reinterpret_cast<uint4*>(chunk);
    for (int i = tid; i < 4 * KS * 2 * 32; i += 128) {
        const int ln = i & 31, g = ln >> 2, t = ln & 3, two = i >> 5 & 1, ks = (i >> 6) % KS, cg = (i >> 6) / KS;
        const int ch = cg * (D / 4) + ks * 16 + 2 * t;
        const float* src = (two ? q_s : kg_s) + g * DC_LD + ch;
        uint32_t p[3][4];
#pragma unroll
        for (int tile = 0; tile < 2; ++tile)
#pragma unroll
            for (int b = 0; b < 2; ++b) {
                const float2 v = *reinterpret_cast<const float2*>(src + tile * 8 * DC_LD + b * 8);
                t5_split3(v.x, v.y, p[0][2 * tile + b], p[1][2 * tile + b], p[2][2 * tile + b]);
            }
#pragma unroll
        for (int j = 0; j < 3; ++j) fa[((i >> 5) * 3 + j) * 32 + ln] = make_uint4(p[j][0], p[j][1], p[j][2], p[j][3]);
    }
    // of KE: item (group of channels, 16 of its channels, lane)
    uint4* fu = reinterpret_cast<uint4*>(chunk + DcChunk<D>::FA);
    for (int i = tid; i < 4 * KS * 32; i += 128) {
        const int ln = i & 31, g = ln >> 2, t = ln & 3, ch = (i >> 5) * 16 + g;
        uint32_t p[3][4];
#pragma unroll
        for (int tile = 0; tile < 2; ++tile)
#pragma unroll
            for (int b = 0; b < 2; ++b) {
                const float* src = ke_s + (2 * t + 8 * b) * DC_LD + ch + tile * 8;
                t5_split3(src[0], src[DC_LD], p[0][2 * tile + b], p[1][2 * tile + b], p[2][2 * tile + b]);
            }
#pragma unroll
        for (int j = 0; j < 3; ++j) fu[((i >> 5) * 3 + j) * 32 + ln] = make_uint4(p[j][0], p[j][1], p[j][2], p[j][3]);
    }
    // of B
    if (tid >= 32 && tid < 32 + DC_T) reinterpret_cast<float*>(chunk + DcChunk<D>::AT_BD)[tid - 32] = diag_s[tid - 32];
    if (tid < 32) {
        uint4* fb = reinterpret_cast<uint4*>(chunk + DcChunk<D>::FA + DcChunk<D>::FU);
        const int g = lane >> 2, t = lane & 3;
        uint32_t p[3][4];
#pragma unroll
        for (int tile = 0; tile < 2; ++tile)
#pragma unroll
            for (int b = 0; b < 2; ++b)
                t5_split3(B_s[tile * 8 + g][2 * t + 8 * b], B_s[tile * 8 + g][2 * t + 8 * b + 1], p[0][2 * tile + b], p[1][2 * tile + b], p[2][2 * tile + b]);
#pragma unroll
        for (int j = 0; j < 3; ++j) fb[j * 32 + lane] = make_uint4(p[j][0], p[j][1], p[j][2], p[j][3]);
    }
}

__device__ __forceinline__ void dc_mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void dc_bulk(void* dst, const void* src, int bytes, void* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(t5_smem(dst)), "l"(src), "r"(bytes), "r"(t5_smem(bar)) : "memory");
}

// B u of a chunk by multiply-adds over the tokens in front of an output's own, where an update is not finite: the tensor core multiplies it
// with the zeros that B has for the tokens in front of it, and would make NaN of their outputs.  w: a lane's updates as the walk has them;
// fb: B's fragments (three parts of 32 lanes' four words).  By a whole warp.
__device__ __forceinline__ void dc_outputs_in_order(const float (&w)[8], const uint32_t* fb, int g, int t, float (&acc)[2][4]) {
#pragma unroll
    for (int e = 0; e < 8; ++e) acc[e / 4][e % 4] = 0.f;
#pragma unroll
    for (int s = 0; s < DC_T; ++s) {
        const int from = s % 8 / 2;                          // the lane of column g that has token s, and B's of token s in a row
        const float lo = __shfl_sync(0xffffffffu, w[s / 8 * 4 + s % 2], g * 4 + from), hi = __shfl_sync(0xffffffffu, w[s / 8 * 4 + 2 + s % 2], g * 4 + from);
#pragma unroll
        for (int tile = 0; tile < 2; ++tile)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int row = 2 * t + e;
                float b = 0.f;
#pragma unroll
                for (int j = 0; j < 3; ++j) {
                    const uint32_t pair = fb[(j * 32 + row * 4 + from) * 4 + 2 * tile + s / 8];
                    b += __uint_as_float(s % 2 ? pair & 0xffff0000u : pair << 16);
                }
                if (s < tile * 8 + row) {
                    acc[tile][e] = fmaf(lo, b, acc[tile][e]);
                    acc[tile][2 + e] = fmaf(hi, b, acc[tile][2 + e]);
                }
            }
    }
}

// 16 value columns to a block; four warps share the channels, a fifth makes the outputs while they are at the next chunk, and
// waits for the copies so that they need not.  A thread's part of the state: columns g and g + 8 (rows of the tensor core's
// tiles), of each of TN tiles the channels 2 t and 2 t + 1, where g and t are the lane's quotient and rest by 4.
// 32 columns to a block, with two sets of warps that read the same operands, take 197 us for 2,048 tokens where 16 take 105: what
// bounds a chunk is the reading of its operands from shared memory and the chain split - products - sums - products.
template <int D>
__global__ void __launch_bounds__(160, 1)
delta_chunk_walk_kernel(const unsigned char* __restrict__ chunks, float* __restrict__ state, long long state_stride, const int* __restrict__ spans,
                        float* __restrict__ out, int H, int dv, int row0, int row1, int* __restrict__ error_flag) {
    gi_pdl_start();
    using C = DcChunk<D>;
    constexpr int KS = D / 64, TN = D / 32, STAGE = C::HEAD + DC_COLS * DC_T * 4;
    extern __shared__ __align__(128) unsigned char dw_smem[];                     // stages, then the sums of the four warps, twice
    __shared__ unsigned long long full[DC_STAGES];
    __shared__ int gave_up[2];                               // by the parity of the chunk whose barrier tells it
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const int h = blockIdx.y, v0 = blockIdx.z * DC_COLS, cg = warp;
    const DcSpan sp = dc_span(spans, blockIdx.x, row0, row1);
    if (sp.len <= 0) return;
    if (sp.slot < 0) {
        for (int i = tid; i < sp.len * DC_COLS; i += 160) out[(size_t)(sp.start + i / DC_COLS) * H * dv + h * dv + v0 + i % DC_COLS] = 0.f;
        return;
    }
    const int n = (sp.len + DC_T - 1) / DC_T;
    const size_t chunk_bytes = C::HEAD + (size_t)DC_T * 4 * dv;
    const unsigned char* src = chunks + ((size_t)sp.chunk0 * H + h) * chunk_bytes;
    float4* sums = reinterpret_cast<float4*>(dw_smem + DC_STAGES * STAGE);        // [2][4 warps][4][32]
    auto total = [&](int c, int i) {                         // of the four warps, in order
        const float4* x = sums + (c & 1) * 512 + i * 32 + lane;
        const float4 a = x[0], b = x[128], d = x[256], e = x[384];
        return make_float4(((a.x + b.x) + d.x) + e.x, ((a.y + b.y) + d.y) + e.y, ((a.z + b.z) + d.z) + e.z, ((a.w + b.w) + d.w) + e.w);
    };
    // u of columns g, g + 8 and tokens 2 t, 2 t + 1 (first tile of rows) and 8 later: the tensor core's first operand
    auto updates = [&](int c, const float4& lo, const float4& hi, float (&w)[8]) {
        const float4 s0 = total(c, 0), s1 = total(c, 1);
        w[0] = lo.x - s0.x; w[1] = lo.y - s0.y; w[2] = hi.x - s0.z; w[3] = hi.y - s0.w;
        w[4] = lo.z - s1.x; w[5] = lo.w - s1.y; w[6] = hi.z - s1.z; w[7] = hi.w - s1.w;
    };
    auto parts = [](const float (&w)[8], uint32_t (&u)[3][4]) {
#pragma unroll
        for (int i = 0; i < 4; ++i) t5_split3(w[2 * i], w[2 * i + 1], u[0][i], u[1][i], u[2][i]);
    };
    constexpr int OF_A[6] = {2, 0, 1, 1, 0, 0}, OF_B[6] = {0, 2, 1, 0, 1, 0};      // small products first, the last one large

    if (warp == 4) {
        auto fetch = [&](int c) {
            const int s = c % DC_STAGES;
            const unsigned char* from = src + (size_t)c * H * chunk_bytes;
            t5_bar_expect(&full[s], STAGE);
            dc_bulk(dw_smem + s * STAGE, from, C::HEAD, &full[s]);
            dc_bulk(dw_smem + s * STAGE + C::HEAD, from + C::HEAD + (size_t)v0 * DC_T * 4, DC_COLS * DC_T * 4, &full[s]);
        };
        // chunk c's copies have landed when the barrier of chunk c - 1 lets go
        auto arrived = [&](int c) {
            if (lane == 0 && c < n) {
                int never = 0;
                if (!t5_bar_wait(&full[c % DC_STAGES], c / DC_STAGES & 1, &never)) gave_up[c & 1] = 1;
            }
            __syncwarp();
        };
        if (lane == 0) {
            for (int s = 0; s < DC_STAGES; ++s) t5_bar_init(&full[s], 1);
            gave_up[0] = gave_up[1] = 0;
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
            for (int c = 0; c < min(n, DC_STAGES); ++c) fetch(c);
        }
        __syncwarp();
        arrived(0);
        __syncthreads();
        bool ok = !gave_up[0];
        for (int c = 0; c < n && ok; ++c) {
            arrived(c + 1);
            __syncthreads();                                 // the sums of this chunk are there, and its stage's predecessor is done with
            ok = !gave_up[(c + 1) & 1];
            if (lane == 0 && c > 0 && c - 1 + DC_STAGES < n) fetch(c - 1 + DC_STAGES);
            const unsigned char* stage = dw_smem + c % DC_STAGES * STAGE;
            const float4* tv = reinterpret_cast<const float4*>(stage + C::HEAD) + lane * 2;
            float w[8];
            updates(c, tv[0], tv[1], w);
            const uint4* fb = reinterpret_cast<const uint4*>(stage + C::FA + C::FU) + lane;
            const uint4 b[3] = {fb[0], fb[32], fb[64]};
            const float2* diag = reinterpret_cast<const float2*>(stage + C::AT_BD) + t;
            const float2 own[2] = {diag[0], diag[4]};
            const float4 of_state[2] = {total(c, 2), total(c, 3)};
            uint32_t u[3][4];
            parts(w, u);
            float acc[2][4] = {}, large[2][4] = {};
#pragma unroll
            for (int m = 0; m < 6; ++m) {
                dc_mma(m == 5 ? large[0] : acc[0], u[OF_A[m]], b[OF_B[m]].x, b[OF_B[m]].y);
                dc_mma(m == 5 ? large[1] : acc[1], u[OF_A[m]], b[OF_B[m]].z, b[OF_B[m]].w);
            }
            float zero[2] = {0.f, 0.f};                      // NaN where a sum is not finite
#pragma unroll
            for (int tile = 0; tile < 2; ++tile)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    acc[tile][e] += large[tile][e];
                    zero[tile] = fmaf(acc[tile][e], 0.f, zero[tile]);
                }
            if (__builtin_expect(__any_sync(0xffffffffu, zero[0] + zero[1] != 0.f), 0))
                dc_outputs_in_order(w, reinterpret_cast<const uint32_t*>(fb - lane), g, t, acc);
#pragma unroll
            for (int tile = 0; tile < 2; ++tile) {
                const float4 s = of_state[tile];
                const float2 b1 = own[tile];
                const int at = c * DC_T + tile * 8 + 2 * t;
                float* dst = out + (size_t)(sp.start + at) * H * dv + h * dv + v0 + g;
                if (at < sp.len) { dst[0] = fmaf(b1.x, w[tile * 4], acc[tile][0] + s.x); dst[8] = fmaf(b1.x, w[tile * 4 + 2], acc[tile][2] + s.z); }
                if (at + 1 < sp.len) {
                    dst[(size_t)H * dv] = fmaf(b1.y, w[tile * 4 + 1], acc[tile][1] + s.y);
                    dst[(size_t)H * dv + 8] = fmaf(b1.y, w[tile * 4 + 3], acc[tile][3] + s.w);
                }
            }
        }
        if (!ok && lane == 0) {                     // the copies still in flight land before the block leaves
            atomicExch(error_flag, DC_ERR_WAIT);
            int never = 0;
            for (int s = 0; s < min(n, DC_STAGES); ++s) {
                t5_bar_wait(&full[s], 0, &never);
                t5_bar_wait(&full[s], 1, &never);
            }
        }
        return;
    }

    float S[TN][4];
    float* st = state + (size_t)sp.slot * state_stride + ((size_t)h * dv + v0 + g) * D + cg * (D / 4) + 2 * t;
#pragma unroll
    for (int i = 0; i < TN; ++i) {
        const float2 lo = *reinterpret_cast<const float2*>(st + i * 8), hi = *reinterpret_cast<const float2*>(st + (size_t)8 * D + i * 8);
        S[i][0] = lo.x; S[i][1] = lo.y; S[i][2] = hi.x; S[i][3] = hi.y;
    }
    __syncthreads();
    if (gave_up[0]) return;
    uint4 fa[KS][2][3];                                      // the rows' fragments of the chunk that is next
    auto rows_of = [&](int c) {
        const uint4* p = reinterpret_cast<const uint4*>(dw_smem + c % DC_STAGES * STAGE) + (size_t)cg * KS * 6 * 32 + lane;
#pragma unroll
        for (int i = 0; i < KS * 6; ++i) fa[i / 6][i / 3 % 2][i % 3] = p[i * 32];
    };
    rows_of(0);
    for (int c = 0; c < n; ++c) {
        const unsigned char* stage = dw_smem + c % DC_STAGES * STAGE;
        uint4 b[KS][3];
        float4 lo, hi;
        float2 decay[TN];
        {   // the rows [T KG; QG] times the state, this warp's channels: chains of at most six products, side by side
            float small[KS][4][4], large[4][4];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    large[i][e] = 0.f;
#pragma unroll
                    for (int ks = 0; ks < KS; ++ks) small[ks][i][e] = 0.f;
                }
#pragma unroll
            for (int ks = 0; ks < KS; ++ks) {
                uint32_t a[3][4];
#pragma unroll
                for (int j = 0; j < 2; ++j)
#pragma unroll
                    for (int r = 0; r < 2; ++r)
                        t5_split3(S[2 * ks + j][2 * r], S[2 * ks + j][2 * r + 1], a[0][2 * j + r], a[1][2 * j + r], a[2][2 * j + r]);
#pragma unroll
                for (int m = 0; m < 6; ++m)
#pragma unroll
                    for (int two = 0; two < 2; ++two) {
                        const uint4 w = fa[ks][two][OF_B[m]];
                        dc_mma(m == 5 ? large[2 * two] : small[ks][2 * two], a[OF_A[m]], w.x, w.y);
                        dc_mma(m == 5 ? large[2 * two + 1] : small[ks][2 * two + 1], a[OF_A[m]], w.z, w.w);
                    }
            }
            // (what the other half of the step reads of the chunk is on its way before the barrier)
            const uint4* fu = reinterpret_cast<const uint4*>(stage + C::FA) + (size_t)cg * KS * 3 * 32 + lane;
            const float4* tv = reinterpret_cast<const float4*>(stage + C::HEAD) + lane * 2;
            const float* G = reinterpret_cast<const float*>(stage + C::AT_G) + cg * (D / 4) + 2 * t;
            lo = tv[0];
            hi = tv[1];
#pragma unroll
            for (int i = 0; i < KS * 3; ++i) b[i / 3][i % 3] = fu[i * 32];
#pragma unroll
            for (int i = 0; i < TN; ++i) decay[i] = *reinterpret_cast<const float2*>(G + i * 8);
            float4* mine = sums + (c & 1) * 512 + cg * 128 + lane;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                float x[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) x[e] = large[i][e] + (KS == 2 ? small[0][i][e] + small[KS - 1][i][e] : small[0][i][e]);
                mine[i * 32] = make_float4(x[0], x[1], x[2], x[3]);
            }
        }
        __syncthreads();
        if (gave_up[(c + 1) & 1]) return;
        uint32_t u[3][4];
        float last[2];                                       // the last token's updates of columns g and g + 8, and its key
        float2 key[TN];
        {
            float w[8];
            updates(c, lo, hi, w);
            parts(w, u);
            const float* K = reinterpret_cast<const float*>(stage + C::AT_KL) + cg * (D / 4) + 2 * t;
#pragma unroll
            for (int i = 0; i < TN; ++i) key[i] = *reinterpret_cast<const float2*>(K + i * 8);
            const int at = min(DC_T, sp.len - c * DC_T) - 1, from = g * 4 + at % 8 / 2;
            const float even[2] = {at < 8 ? w[0] : w[4], at < 8 ? w[2] : w[6]}, odd[2] = {at < 8 ? w[1] : w[5], at < 8 ? w[3] : w[7]};
#pragma unroll
            for (int i = 0; i < 2; ++i) last[i] = __shfl_sync(0xffffffffu, at % 2 ? odd[i] : even[i], from);
        }
        float small[TN][4], large[TN][4];
#pragma unroll
        for (int i = 0; i < TN; ++i)
#pragma unroll
            for (int e = 0; e < 4; ++e) small[i][e] = large[i][e] = 0.f;
#pragma unroll
        for (int m = 0; m < 6; ++m)
#pragma unroll
            for (int ks = 0; ks < KS; ++ks) {
                const uint4 w = b[ks][OF_B[m]];
                dc_mma(m == 5 ? large[2 * ks] : small[2 * ks], u[OF_A[m]], w.x, w.y);
                dc_mma(m == 5 ? large[2 * ks + 1] : small[2 * ks + 1], u[OF_A[m]], w.z, w.w);
            }
#pragma unroll
        for (int i = 0; i < TN; ++i) {
#pragma unroll
            for (int e = 0; e < 4; ++e)
                S[i][e] = fmaf(last[e >> 1], e & 1 ? key[i].y : key[i].x, fmaf(S[i][e], e & 1 ? decay[i].y : decay[i].x, small[i][e] + large[i][e]));
        }
        if (c + 1 < n) rows_of(c + 1);
    }
#pragma unroll
    for (int i = 0; i < TN; ++i) {
        *reinterpret_cast<float2*>(st + i * 8) = make_float2(S[i][0], S[i][1]);
        *reinterpret_cast<float2*>(st + (size_t)8 * D + i * 8) = make_float2(S[i][2], S[i][3]);
    }
}

// bytes that a chunk (16 tokens of one sequence at most) takes, all heads
extern "C" long long gi_delta_chunk_bytes(int H, int d, int dv) {
    return (long long)H * ((d == 128 ? DcChunk<128>::HEAD : DcChunk<64>::HEAD) + DC_T * 4LL * dv);
}

template <int D, int CH>
static int launch_delta_chunk(const float* qkv, long long ldq, int q_off, int k_off, int v_off, const float* ab, long long ldab, int b_off,
                              int a_off, const float* al, long long ldal, const void* A_log, const void* dt_bias, int p_dtype, float* state,
                              long long state_stride, const int* spans, float* out, unsigned char* space, int rows_at_a_time, int n_rows, int n_seq,
                              int H, int Hk, int dv, float unit_eps, float q_scale, int* error_flag, cudaStream_t s) {
    const auto prepare = delta_chunk_prepare_kernel<D, CH>;
    const auto walk = delta_chunk_walk_kernel<D>;
    const size_t smem_p = 5 * DC_T * DC_LD * sizeof(float);
    const size_t smem_w = (size_t)DC_STAGES * (DcChunk<D>::HEAD + DC_COLS * DC_T * 4) + 2 * 512 * sizeof(float4);
    if (int rc = gi_reserve_smem((const void*)prepare, smem_p, "gi_delta_chunk_scan")) return rc;
    if (int rc = gi_reserve_smem((const void*)walk, smem_w, "gi_delta_chunk_scan")) return rc;
    for (long long row0 = 0; row0 < n_rows; row0 += rows_at_a_time) {
        const int rows = (int)(n_rows - row0 < rows_at_a_time ? n_rows - row0 : rows_at_a_time);
        gi_launch(prepare, dim3(rows / DC_T + n_seq, H), dim3(128), smem_p, s, qkv, ldq, q_off, k_off, v_off, ab, ldab, b_off, a_off, al, ldal, A_log,
                  dt_bias, p_dtype, spans, n_seq, space, H, Hk, dv, unit_eps, q_scale, (int)row0, (int)row0 + rows);
        if (int rc = gi_check_launch("gi_delta_chunk_scan")) return rc;
        gi_launch(walk, dim3(n_seq, H, dv / DC_COLS), dim3(160), smem_w, s, (const unsigned char*)space, state, state_stride, spans, out, H, dv,
                  (int)row0, (int)row0 + rows, error_flag);
        if (int rc = gi_check_launch("gi_delta_chunk_scan")) return rc;
    }
    return 0;
}

// The arguments of gi_delta_scan_prompt; space: (rows_at_a_time / 16 + n_seq) gi_delta_chunk_bytes, on 16 bytes.
extern "C" int gi_delta_chunk_scan(const float* qkv, long long ldq, int q_off, int k_off, int v_off, const float* ab, long long ldab, int b_off,
                                   int a_off, const float* a_sep, long long lda_sep, const void* A_log, const void* dt_bias, int p_dtype,
                                   float* state, long long state_stride, const int* spans, float* out, void* space, int rows_at_a_time,
                                   int n_rows, int n_seq, int H, int Hk, int d, int dv, float unit_eps, float q_scale, int channel_decay,
                                   int* error_flag, void* stream) {
    GI_REQUIRE(n_seq >= 0 && n_rows >= 0 && H > 0 && Hk > 0 && H % Hk == 0 && (d == 64 || d == 128) && dv > 0 && dv % DC_COLS == 0,
               "gi_delta_chunk_scan: %d heads on %d key heads, keys of %d, values of %d", H, Hk, d, dv);
    GI_REQUIRE(H <= 65535 && dv / DC_COLS <= 65535, "gi_delta_chunk_scan: %d heads of %d values", H, dv);
    GI_REQUIRE(state_stride >= (long long)H * dv * d && state_stride % 4 == 0 && (uintptr_t)state % 16 == 0,
               "gi_delta_chunk_scan: state rows of %lld floats", state_stride);
    GI_REQUIRE(ldq % 4 == 0 && q_off % 4 == 0 && k_off % 4 == 0 && ((uintptr_t)qkv | (uintptr_t)space) % 16 == 0,
               "gi_delta_chunk_scan: rows start on 16 bytes");
    GI_REQUIRE(rows_at_a_time > 0 && error_flag, "gi_delta_chunk_scan: room for %d rows, an error flag", rows_at_a_time);
    if (n_seq == 0 || n_rows == 0) return 0;
    const float* al = a_sep ? a_sep : ab;
    const long long ldal = a_sep ? lda_sep : ldab;
#define DC_GO(D, CH) launch_delta_chunk<D, CH>(qkv, ldq, q_off, k_off, v_off, ab, ldab, b_off, a_off, al, ldal, A_log, dt_bias, p_dtype, state, \
        state_stride, spans, out, (unsigned char*)space, rows_at_a_time, n_rows, n_seq, H, Hk, dv, unit_eps, q_scale, error_flag, (cudaStream_t)stream)
    if (d == 128) return channel_decay ? DC_GO(128, 1) : DC_GO(128, 0);
    return channel_decay ? DC_GO(64, 1) : DC_GO(64, 0);
#undef DC_GO
}
