// Mixers that carry a matrix of state per head from token to token, and the short causal convolution in
// front of one of them.  All state is float32 and lives in the cache's per-slot state rows.
//
//   gi_causal_conv_silu     y[t, c] = silu( sum_j taps[c, j] x[t - (K-1) + j, c] ), zeros before position 0; the
//                           K-1 inputs before this step's first token come from the slot's state
//   gi_conv_state_update    afterwards: the slot's state becomes its last K-1 inputs
//   gi_decay_scan           S_t = lam_h S_(t-1) + k_t v_t^T,  o_t = S_t^T q_t           (q, k, v = silu of the
//                           projections): linear attention with one fixed decay per head
//   gi_delta_scan           S <- g_t S;  u = beta_t (v_t - S^T k_t);  S <- S + k_t u^T;  o_t = S^T q_t
//                           with q, k made unit vectors per head (q also times dim^-1/2),
//                           g_t = exp(-exp(A_h) softplus(a_t + dt_h)),  beta_t = sigmoid(b_t): the gated delta rule;
//                           the decay is one number per head, or one per head and key channel (row c of a head's
//                           state times g_t[c])
//
// A scan block owns one (sequence, head, slice of 32 value columns) and walks the sequence's tokens of this
// step in order, so prompts, portions of prompts and single tokens run the same instructions in the same
// order and give the same bits.  P lanes share one value column: a thread holds R of the column's keys in
// registers (4 consecutive keys out of every 4 P), and sums over the keys end with log2(P) shuffles.  P is 4 or
// 8 by the key dimension alone (8 from 64 keys on): with one long prompt there are only heads x columns / 32
// blocks, and it is the warps of a block that hide each other's latencies.  Measured at keys of 128, 32 heads
// (P = 4 / 8 / 16): a prompt of 2,048 tokens 0.91 / 0.71 / 0.70 ms (decay) and 1.61 / 1.23 / 1.04 ms (delta rule); a
// whole decode step of 64 sequences 1.72 / 1.80 / 1.89 ms.  P never depends on the batch or the cut, so a
// position's bits do not either.
// The delta rule's scan asks for the next chunk's inputs (into registers) before it walks the present chunk's
// tokens, when the rows allow 16-byte loads: a prompt of 2,048 tokens, 16 heads of 128 x 128, 1.20 -> 0.77 ms with a
// decay per head and 1.68 -> 1.07 ms with one per key channel; what is computed, and in which order, is the same.
// State rows are laid out [head][value column][key, padded to R P] so that a warp's loads and stores are
// whole runs of 16 P bytes.  NikolayBlagoev/garlic-inference has no recurrent mixer.
#include "scan.cuh"

// ------------------------------------------------------------------ short causal convolution
#define CONV_MAX_TAPS 16

// In-step predecessors of row r that belong to the same sequence, at most `most`.
__device__ __forceinline__ int rows_before(const int* __restrict__ tok_slot, int r, int slot, int most) {
    int have = 0;
    while (have < most && r - have - 1 >= 0 && tok_slot[r - have - 1] == slot) ++have;
    return have;
}

template <typename T>
__global__ void causal_conv_silu_kernel(const T* __restrict__ x, long long ldx, int C, const void* __restrict__ taps,
                                        int taps_dtype, int K, const float* __restrict__ state, long long state_stride,
                                        const int* __restrict__ tok_slot, float* __restrict__ out, int act,
                                        float* __restrict__ state_out, const void* __restrict__ in_bias,
                                        const void* __restrict__ out_bias, int bias_dtype) {
    gi_pdl_start();
    const int r = blockIdx.x;
    const int c = blockIdx.y * blockDim.x + threadIdx.x;
    if (c >= C) return;
    const int slot = tok_slot[r];
    const int have = slot < 0 ? 0 : rows_before(tok_slot, r, slot, K - 1);
    // a bias on the inputs belongs to the tokens (what the state holds has it already, and before a sequence's
    // first token there are zeros, not biases); a bias on the outputs starts the sum
    const float bin = in_bias ? load_w(in_bias, bias_dtype, c) : 0.f;
    float acc = out_bias ? load_w(out_bias, bias_dtype, c) : 0.f;
    float seen[CONV_MAX_TAPS];                       // the inputs, oldest first (for the state when it is renewed here)
    for (int j = K - 1; j >= 0; --j) {               // oldest input first, whatever its source
        float xv = 0.f;
        if (j <= have) xv = to_f32(x[(size_t)(r - j) * ldx + c]) + bin;
        else if (slot >= 0) xv = state[(size_t)slot * state_stride + (size_t)(K - 1 + have - j) * C + c];
        seen[K - 1 - j] = xv;
        acc = fmaf(load_w(taps, taps_dtype, c * K + (K - 1 - j)), xv, acc);
    }
    out[(size_t)r * C + c] = act ? rc_silu(acc) : acc;
    // Steps in which every row is a sequence of its own (decode steps): the slot's state becomes its last K - 1 inputs
    // here, by the one thread that read it, instead of in a launch of its own.
    if (state_out && slot >= 0)
        for (int m = 0; m < K - 1; ++m) state_out[(size_t)slot * state_stride + (size_t)m * C + c] = seen[m + 1];
}

// The same filter for prompts: a thread keeps CONV_V neighbouring channels of CONV_ROWS rows, the K - 1 inputs before a
// row in registers, so that every input is fetched once (and K - 1 of CONV_ROWS + K - 1 rows once more by the
// neighbour) instead of K times one element at a time.  Bound by memory: it reads 2 and writes 4 bytes an element.
// Measured at 2,048 rows of 4,096 bfloat16 channels and 4 taps: 73 us with a thread per element, 21 us so.  The
// order of a sum is the other kernel's, oldest input first, and so are the bits.  Taken for up to 4 taps (beyond, the
// window's registers pass what a vector of channels gains) where channels come in whole aligned vectors and the step has
// enough elements that its threads fill the chip (a thread has 32): per element / in rows in us at 4,096 channels 34 rows 3.8 / 8.3,
// 64 rows 4.1 / 5.7, 256 rows 10.6 / 6.9; 512 channels 1,024 rows 6.4 / 7.2.
#define CONV_MIN_ELEMENTS (3LL << 18)
#define CONV_ROWS 8
#define CONV_V 4
template <typename T, int K>
__global__ void __launch_bounds__(128)
causal_conv_rows_kernel(const T* __restrict__ x, long long ldx, int C, const void* __restrict__ taps, int taps_dtype,
                        const float* __restrict__ state, long long state_stride, const int* __restrict__ tok_slot,
                        float* __restrict__ out, int n_rows, int act, const void* __restrict__ in_bias,
                        const void* __restrict__ out_bias, int bias_dtype) {
    gi_pdl_start();
    const int r0 = blockIdx.x * CONV_ROWS, c = (blockIdx.y * blockDim.x + threadIdx.x) * CONV_V;
    if (c >= C) return;
    float w[CONV_V][K], bin[CONV_V], bout[CONV_V];
#pragma unroll
    for (int v = 0; v < CONV_V; ++v) {
#pragma unroll
        for (int j = 0; j < K; ++j) w[v][j] = load_w(taps, taps_dtype, (c + v) * K + j);
        bin[v] = in_bias ? load_w(in_bias, bias_dtype, c + v) : 0.f;
        bout[v] = out_bias ? load_w(out_bias, bias_dtype, c + v) : 0.f;
    }
    float4 in[CONV_ROWS + K - 1];                    // rows r0 - (K - 1) .. r0 + CONV_ROWS - 1, with the tokens' bias
    int slots[CONV_ROWS + K - 1];
#pragma unroll
    for (int i = 0; i < CONV_ROWS + K - 1; ++i) {
        const int r = min(max(r0 - (K - 1) + i, 0), n_rows - 1);
        in[i] = load4_act(x + (size_t)r * ldx + c);
        slots[i] = r0 - (K - 1) + i < 0 ? -1 : tok_slot[r];
    }
#pragma unroll
    for (int i = 0; i < CONV_ROWS + K - 1; ++i) { in[i].x += bin[0]; in[i].y += bin[1]; in[i].z += bin[2]; in[i].w += bin[3]; }
#pragma unroll
    for (int i = 0; i < CONV_ROWS; ++i) {
        const int r = r0 + i, at = i + K - 1;
        if (r >= n_rows) break;
        const int slot = slots[at];
        int have = 0;                                // rows right before this one of the same sequence
        bool same = slot >= 0;
#pragma unroll
        for (int j = 1; j < K; ++j) {
            same = same && slots[at - j] == slot;
            have += same;
        }
        float4 acc = make_float4(bout[0], bout[1], bout[2], bout[3]);
#pragma unroll
        for (int j = K - 1; j >= 0; --j) {
            float4 xv = in[at - j];
            if (j > have) {
                xv = make_float4(0.f, 0.f, 0.f, 0.f);
                if (slot >= 0) {
                    const float* st = state + (size_t)slot * state_stride + (size_t)(K - 1 + have - j) * C + c;
                    xv = make_float4(st[0], st[1], st[2], st[3]);
                }
            }
            acc.x = fmaf(w[0][K - 1 - j], xv.x, acc.x);
            acc.y = fmaf(w[1][K - 1 - j], xv.y, acc.y);
            acc.z = fmaf(w[2][K - 1 - j], xv.z, acc.z);
            acc.w = fmaf(w[3][K - 1 - j], xv.w, acc.w);
        }
        if (act) acc = make_float4(rc_silu(acc.x), rc_silu(acc.y), rc_silu(acc.z), rc_silu(acc.w));
        *reinterpret_cast<float4*>(out + (size_t)r * C + c) = acc;
    }
}

// A block looks through `span` rows (at most 32) for the last ones of sequences; its eight warps take them in turn and renew
// CONV_STATE_C channels of their slots' states.  KK: the taps, 0: as many as are asked for.  What is read is asked for before
// any of it is looked at: a warp's time is two trips to memory (the slots, then the inputs).  4,096 channels in us, a block per
// row and 128 channels / a block that renewed one last row of 32 after the other / so: one prompt of 2,048 68 / 4.5 / 3.5 (the
// first is the launching of 65,536 blocks), 512 sequences of 2 tokens 35 / 57 / 9, 33 of 1 and one of 20 3.2 / 90 / 2.9.
#define CONV_STATE_C 256
template <typename T, int KK>
__global__ void __launch_bounds__(256)
conv_state_update_kernel(const T* __restrict__ x, long long ldx, int C, int K_,
                         float* __restrict__ state, long long state_stride,
                         const int* __restrict__ tok_slot, int n_rows, int span,
                         const void* __restrict__ in_bias, int bias_dtype) {
    gi_pdl_start();
    constexpr int PER = CONV_STATE_C / 32, KEEP = (KK ? KK : CONV_MAX_TAPS) - 1, AT_ONCE = KK ? PER : 1;
    const int K = KK ? KK : K_, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, row = blockIdx.x * span + lane;
    const bool in = lane < span && row < n_rows;
    const int own = in ? tok_slot[row] : -1, next = in && row + 1 < n_rows ? tok_slot[row + 1] : -1;
    unsigned last = __ballot_sync(0xffffffffu, own >= 0 && own != next);
    const int c0 = blockIdx.y * CONV_STATE_C + lane;
    for (int nth = 0; last; ++nth, last &= last - 1) {
        if ((nth & 7) != warp) continue;
        const int at = __ffs(last) - 1, r = blockIdx.x * span + at, slot = __shfl_sync(0xffffffffu, own, at);
        const int have = rows_before(tok_slot, r, slot, K - 1);
        float* st = state + (size_t)slot * state_stride;
        for (int i0 = 0; i0 < PER; i0 += AT_ONCE) {          // channels whose inputs are under way together
            float vals[AT_ONCE][KEEP];
            T xs[AT_ONCE][KEEP];
#pragma unroll
            for (int m = 0; m < KEEP; ++m) {                 // a place takes the row K - 2 - m before the last one, or what the state
                if (m >= K - 1) break;                       // held of that age
                const int j = K - 2 - m;
#pragma unroll
                for (int i = 0; i < AT_ONCE; ++i) {
                    const int c = c0 + 32 * (i0 + i);
                    if (c < C) xs[i][m] = x[(size_t)(r - min(j, have)) * ldx + c];
                    if (c < C && have < K - 2) vals[i][m] = st[(size_t)min(K - 1 + have - j, K - 2) * C + c];
                }
            }
#pragma unroll
            for (int i = 0; i < AT_ONCE; ++i) {
                const int c = c0 + 32 * (i0 + i);
                const float bin = in_bias && c < C ? load_w(in_bias, bias_dtype, c) : 0.f;
#pragma unroll
                for (int m = 0; m < KEEP; ++m) {
                    if (m >= K - 1) break;
                    if (K - 2 - m <= have) vals[i][m] = to_f32(xs[i][m]) + bin;
                }
#pragma unroll
                for (int m = 0; m < KEEP; ++m)
                    if (m < K - 1 && c < C) st[(size_t)m * C + c] = vals[i][m];
            }
        }
    }
}

template <typename T>
static bool launch_conv_rows(const T* x, long long ldx, int C, const void* taps, int taps_dtype, int K, const float* state,
                             long long state_stride, const int* tok_slot, float* out, int n_rows, int act,
                             const void* in_bias, const void* out_bias, int bias_dtype, cudaStream_t s) {
    if (K > 4 || (long long)n_rows * C < CONV_MIN_ELEMENTS || C % CONV_V || ldx % CONV_V || (uintptr_t)x % (CONV_V * sizeof(T)) || (uintptr_t)out % 16)
        return false;
    dim3 grid((n_rows + CONV_ROWS - 1) / CONV_ROWS, (C + 128 * CONV_V - 1) / (128 * CONV_V));
#define CONV_LAUNCH(KK)                                                                                                       \
    case KK: gi_launch(causal_conv_rows_kernel<T, KK>, grid, dim3(128), 0, s, x, ldx, C, taps, taps_dtype, state, state_stride, \
                       tok_slot, out, n_rows, act, in_bias, out_bias, bias_dtype); break;
    switch (K) { CONV_LAUNCH(1) CONV_LAUNCH(2) CONV_LAUNCH(3) CONV_LAUNCH(4) }
#undef CONV_LAUNCH
    return true;
}

template <typename T>
static void launch_conv(const T* x, long long ldx, int C, const void* taps, int taps_dtype, int K, float* state,
                        long long state_stride, const int* tok_slot, float* out, int n_rows, int update_state, int act,
                        const void* in_bias, const void* out_bias, int bias_dtype, cudaStream_t s) {
    if (update_state == 1) {
        if (K <= 1) return;
        const auto kernel = K == 2 ? conv_state_update_kernel<T, 2> : K == 3 ? conv_state_update_kernel<T, 3> : K == 4 ? conv_state_update_kernel<T, 4> : conv_state_update_kernel<T, 0>;
        // few rows: a warp for each, should they all be last ones; many: fewer blocks (what costs is launching them)
        const int span = n_rows <= 512 ? 8 : 32;
        gi_launch(kernel, dim3((n_rows + span - 1) / span, (C + CONV_STATE_C - 1) / CONV_STATE_C), dim3(256), 0, s, x, ldx, C, K, state,
                  state_stride, tok_slot, n_rows, span, in_bias, bias_dtype);
        return;
    }
    // (a step whose rows are all sequences of their own renews the state in the launch of a thread per element)
    if (update_state == 0 && launch_conv_rows<T>(x, ldx, C, taps, taps_dtype, K, state, state_stride, tok_slot, out, n_rows, act,
                                                 in_bias, out_bias, bias_dtype, s)) return;
    dim3 grid(n_rows, (C + 127) / 128);
    gi_launch(causal_conv_silu_kernel<T>, grid, dim3(128), 0, s, x, ldx, C, taps, taps_dtype, K, (const float*)state, state_stride,
              tok_slot, out, act, update_state == 2 && K > 1 ? state : (float*)nullptr, in_bias, out_bias, bias_dtype);
}

// `act` 1: silu of the filter's sum; 0: the sum itself.  update_state 2: the filter and the renewal of the state in
// one launch, for steps in which no two rows belong to one sequence (the caller's promise).
// `in_bias` (one per channel, added to every input of a token) and `out_bias` (one per channel, added to the sum)
// may be null; they share `bias_dtype`.
extern "C" int gi_causal_conv_biased(const void* x, long long ldx, int act_dtype, int C, const void* taps, int taps_dtype,
                                     int K, float* state, long long state_stride, const int* tok_slot, float* out,
                                     int n_rows, int update_state, int act, const void* in_bias, const void* out_bias,
                                     int bias_dtype, void* stream) {
    GI_REQUIRE(n_rows >= 0 && C > 0 && K >= 1 && K <= CONV_MAX_TAPS, "gi_causal_conv_silu: %d channels, %d taps (1 to %d)",
               C, K, CONV_MAX_TAPS);
    GI_REQUIRE(ldx >= C && state_stride >= (long long)(K - 1) * C, "gi_causal_conv_silu: strides shorter than the rows");
    GI_REQUIRE((C + 127) / 128 <= 65535, "gi_causal_conv_silu: %d channels is beyond %d", C, 65535 * 128);
    if (n_rows == 0) return 0;
    cudaStream_t s = (cudaStream_t)stream;
    if (act_dtype == GI_DTYPE_F32)
        launch_conv<float>((const float*)x, ldx, C, taps, taps_dtype, K, state, state_stride, tok_slot, out, n_rows, update_state, act, in_bias, out_bias, bias_dtype, s);
    else if (act_dtype == GI_DTYPE_BF16)
        launch_conv<bf16>((const bf16*)x, ldx, C, taps, taps_dtype, K, state, state_stride, tok_slot, out, n_rows, update_state, act, in_bias, out_bias, bias_dtype, s);
    else
        GI_REQUIRE(false, "gi_causal_conv_silu: activation dtype %d", act_dtype);
    return gi_check_launch("gi_causal_conv_silu");
}

extern "C" int gi_causal_conv(const void* x, long long ldx, int act_dtype, int C, const void* taps, int taps_dtype,
                              int K, float* state, long long state_stride, const int* tok_slot, float* out,
                              int n_rows, int update_state, int act, void* stream) {
    return gi_causal_conv_biased(x, ldx, act_dtype, C, taps, taps_dtype, K, state, state_stride, tok_slot, out, n_rows,
                                 update_state, act, nullptr, nullptr, GI_DTYPE_F32, stream);
}

extern "C" int gi_causal_conv_silu(const void* x, long long ldx, int act_dtype, int C, const void* taps, int taps_dtype,
                                   int K, float* state, long long state_stride, const int* tok_slot, float* out,
                                   int n_rows, int update_state, void* stream) {
    return gi_causal_conv(x, ldx, act_dtype, C, taps, taps_dtype, K, state, state_stride, tok_slot, out, n_rows,
                          update_state, 1, stream);
}

// ------------------------------------------------------------------ scans (scan.cuh: what they share)
// ---- linear attention with a fixed decay per head
// qkv: T [n, ld], silu applied here; q at column q_off + h d, k at k_off + h d, v at v_off + h dv.
template <typename T, int R, int P>
__global__ void __launch_bounds__(SCAN_VS * P)
decay_scan_kernel(const T* __restrict__ qkv, long long ld, int q_off, int k_off, int v_off,
                  const float* __restrict__ decay, float* __restrict__ state, long long state_stride,
                  const int* __restrict__ spans, const int* __restrict__ tok_slot, float* __restrict__ out,
                  int H, int d, int dv, int vec_rows) {
    gi_pdl_start();
    const bool vec = sizeof(T) == 2 && vec_rows;       // rows that can be fetched 16 bytes at a time
    constexpr int DP = R * P;                          // padded key dimension
    constexpr int TC = SCAN_TC(DP);
    constexpr int SCAN_THREADS = SCAN_VS * P;
    __shared__ __align__(16) float q_s[TC][DP];
    __shared__ __align__(16) float k_s[TC][DP];
    __shared__ float v_s[TC][SCAN_VS];
    __shared__ float o_s[TC][SCAN_VS];
    int slot, start, len;
    scan_span(spans, tok_slot, blockIdx.x, slot, start, len);
    const int h = blockIdx.y, v0 = blockIdx.z * SCAN_VS;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int part = threadIdx.x % P, vl = threadIdx.x / P, v = v0 + vl;
    const bool live = v < dv;
    if (slot < 0) {
        for (int t = 0; t < len; ++t)
            if (live && part == 0) out[(size_t)(start + t) * H * dv + h * dv + v] = 0.f;
        return;
    }
    const float lam = decay[h];
    float* st = state + (size_t)slot * state_stride + ((size_t)h * dv + (live ? v : 0)) * DP;
    float S[R];
    if (live) scan_load_state<R, P>(S, st, part);
    else {
#pragma unroll
        for (int e = 0; e < R; ++e) S[e] = 0.f;
    }
    // Staging.  bfloat16 rows whose heads start on 16 bytes: every thread fetches NV vectors of 8 values of q and
    // k (and one of v) into registers, all at once, and the next chunk's are fetched before this chunk's tokens
    // are walked, so their latency hides behind the walk.  Otherwise: element by element.
    constexpr int VPT = DP / 8;                        // vectors per token and operand
    constexpr int NV = (TC * VPT * 2 + SCAN_THREADS - 1) / SCAN_THREADS;
    uint4 pre[NV], pre_v;
    auto fetch = [&](int t0) {
        const int tc = min(TC, len - t0);
#pragma unroll
        for (int n = 0; n < NV; ++n) {
            const int slot_i = threadIdx.x + SCAN_THREADS * n;
            const int which = slot_i / (TC * VPT), rem = slot_i - which * (TC * VPT);
            const int t = rem / VPT, vc = rem - t * VPT;
            pre[n] = make_uint4(0u, 0u, 0u, 0u);
            if (which < 2 && t < tc && vc * 8 < d)
                pre[n] = *reinterpret_cast<const uint4*>(qkv + (size_t)(start + t0 + t) * ld + (which ? k_off : q_off) + h * d + vc * 8);
        }
        const int t = threadIdx.x / (SCAN_VS / 8), vc = threadIdx.x - t * (SCAN_VS / 8);
        pre_v = make_uint4(0u, 0u, 0u, 0u);
        if (t < tc && v0 + vc * 8 < dv)
            pre_v = *reinterpret_cast<const uint4*>(qkv + (size_t)(start + t0 + t) * ld + v_off + h * dv + v0 + vc * 8);
    };
    auto silu8 = [](const uint4& w, float* dst) {
        const __nv_bfloat162* p2 = reinterpret_cast<const __nv_bfloat162*>(&w);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float2 f = __bfloat1622float2(p2[i]);
            dst[2 * i] = rc_silu(f.x);
            dst[2 * i + 1] = rc_silu(f.y);
        }
    };
    if (vec) fetch(0);
    for (int t0 = 0; t0 < len; t0 += TC) {
        const int tc = min(TC, len - t0);
        __syncthreads();                               // the last chunk's o_s and inputs are done with
        if (vec) {
#pragma unroll
            for (int n = 0; n < NV; ++n) {
                const int slot_i = threadIdx.x + SCAN_THREADS * n;
                const int which = slot_i / (TC * VPT), rem = slot_i - which * (TC * VPT);
                const int t = rem / VPT, vc = rem - t * VPT;
                if (which < 2 && t < tc) silu8(pre[n], (which ? &k_s[t][0] : &q_s[t][0]) + vc * 8);   // silu(0) = 0: the padding
            }
            const int t = threadIdx.x / (SCAN_VS / 8), vc = threadIdx.x - t * (SCAN_VS / 8);
            if (t < tc) silu8(pre_v, &v_s[t][vc * 8]);
        } else {
            for (int i = threadIdx.x; i < tc * DP; i += SCAN_THREADS) {
                const int t = i / DP, c = i - t * DP;
                const T* row = qkv + (size_t)(start + t0 + t) * ld;
                q_s[t][c] = c < d ? rc_silu(to_f32(row[q_off + h * d + c])) : 0.f;
                k_s[t][c] = c < d ? rc_silu(to_f32(row[k_off + h * d + c])) : 0.f;
            }
            for (int i = threadIdx.x; i < tc * SCAN_VS; i += SCAN_THREADS) {
                const int t = i / SCAN_VS, c = i - t * SCAN_VS;
                v_s[t][c] = v0 + c < dv ? rc_silu(to_f32(qkv[(size_t)(start + t0 + t) * ld + v_off + h * dv + v0 + c])) : 0.f;
            }
        }
        __syncthreads();
        if (vec && t0 + TC < len) fetch(t0 + TC);
        for (int t = 0; t < tc; ++t) {
            const float vt = v_s[t][vl];
            float o0 = 0.f, o1 = 0.f, o2 = 0.f, o3 = 0.f;     // four chains instead of one of R dependent steps
#pragma unroll
            for (int i = 0; i < R / 4; ++i) {
                const float4 kk = *reinterpret_cast<const float4*>(&k_s[t][KEY_OF(i, part)]);
                const float4 qq = *reinterpret_cast<const float4*>(&q_s[t][KEY_OF(i, part)]);
                S[4 * i] = fmaf(lam, S[4 * i], kk.x * vt);          o0 = fmaf(S[4 * i], qq.x, o0);
                S[4 * i + 1] = fmaf(lam, S[4 * i + 1], kk.y * vt);  o1 = fmaf(S[4 * i + 1], qq.y, o1);
                S[4 * i + 2] = fmaf(lam, S[4 * i + 2], kk.z * vt);  o2 = fmaf(S[4 * i + 2], qq.z, o2);
                S[4 * i + 3] = fmaf(lam, S[4 * i + 3], kk.w * vt);  o3 = fmaf(S[4 * i + 3], qq.w, o3);
            }
            const float o = part_sum<P>((o0 + o1) + (o2 + o3));
            if (part == 0) o_s[t][vl] = o;
        }
        __syncthreads();
        for (int i = threadIdx.x; i < tc * SCAN_VS; i += SCAN_THREADS) {
            const int t = i / SCAN_VS, c = i - t * SCAN_VS;
            if (v0 + c < dv) out[(size_t)(start + t0 + t) * H * dv + h * dv + v0 + c] = o_s[t][c];
        }
    }
    if (live) scan_store_state<R, P>(S, st, part);
}

// ---- the gated delta rule
// qkv: float32 [n, ldq] (the convolution's output): q of key head kh at q_off + kh d, k at k_off + kh d, v of
// head h at v_off + h dv.  ab: float32 [n, ldab]: beta's logit of head h at column b_off + h, the decay's at
// a_off + h (float32 whatever the activation type is: the decay's logit is multiplied by exp(A_h) and goes
// through two exponentials, which would magnify a 16-bit rounding).
// CH = 1: a decay per head and key channel.  The logits are then [n, H d] (column a_off + h d + c), dt_bias has
// H d elements, and row c of a head's state is multiplied by g[c]; chunks are shorter so that the decays of a
// chunk fit shared memory beside its keys.
#define SCAN_TC_CH(DP) ((DP) <= 64 ? 32 : ((DP) <= 128 ? 16 : 8))
template <typename T, int R, int P, int CH>
__global__ void __launch_bounds__(SCAN_VS * P)
delta_scan_kernel(const float* __restrict__ qkv, long long ldq, int q_off, int k_off, int v_off,
                  const float* __restrict__ ab, long long ldab, int b_off, int a_off,
                  const float* __restrict__ al, long long ldal,
                  const void* __restrict__ A_log, const void* __restrict__ dt_bias, int p_dtype,
                  float* __restrict__ state, long long state_stride, const int* __restrict__ spans,
                  const int* __restrict__ tok_slot, float* __restrict__ out, int H, int Hk, int d, int dv,
                  float unit_eps, float q_scale, int vec) {
    gi_pdl_start();
    constexpr int DP = R * P;
    constexpr int TC = CH ? SCAN_TC_CH(DP) : SCAN_TC(DP);
    constexpr int SCAN_THREADS = SCAN_VS * P;
    __shared__ __align__(16) float q_s[TC][DP];
    __shared__ __align__(16) float k_s[TC][DP];
    __shared__ __align__(16) float gc_s[CH ? TC : 1][CH ? DP : 4];
    __shared__ float v_s[TC][SCAN_VS];
    __shared__ float o_s[TC][SCAN_VS];
    __shared__ float g_s[TC], b_s[TC];
    int slot, start, len;
    scan_span(spans, tok_slot, blockIdx.x, slot, start, len);
    const int h = blockIdx.y, v0 = blockIdx.z * SCAN_VS;
    const int kh = h / (H / Hk);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int part = threadIdx.x % P, vl = threadIdx.x / P, v = v0 + vl;
    const bool live = v < dv;
    if (slot < 0) {
        for (int t = 0; t < len; ++t)
            if (live && part == 0) out[(size_t)(start + t) * H * dv + h * dv + v] = 0.f;
        return;
    }
    const float rate = expf(load_w(A_log, p_dtype, h)), dt = CH ? 0.f : load_w(dt_bias, p_dtype, h);
    float* st = state + (size_t)slot * state_stride + ((size_t)h * dv + (live ? v : 0)) * DP;
    float S[R];
    if (live) scan_load_state<R, P>(S, st, part);
    else {
#pragma unroll
        for (int e = 0; e < R; ++e) S[e] = 0.f;
    }
    // Each warp stages tokens warp, warp + W, ... of a chunk (W warps).  When the rows allow 16-byte loads, the raw
    // values of the NEXT chunk's tokens are asked for into registers before this chunk's tokens are walked, so that
    // the walk hides their latency; what is done with them, and in which order, is the same either way.
    constexpr int TPW = TC / (SCAN_THREADS / 32);
    constexpr int NQ = (DP / 4 + 31) / 32;                 // 16-byte pieces of q (and of k) per lane and token
    constexpr int NA = CH ? (DP + 31) / 32 : 1;            // decay logits per lane and token
    float4 pq[TPW][NQ], pk[TPW][NQ];
    float pv[TPW], pa[TPW][NA], pb[TPW], dtc[NA];
#pragma unroll
    for (int n = 0; n < NA; ++n) {
        const int c = lane + 32 * n;
        dtc[n] = (CH && c < d) ? load_w(dt_bias, p_dtype, h * d + c) : 0.f;
    }
    auto fetch = [&](int t0) {
        const int tc = min(TC, len - t0);
#pragma unroll
        for (int i = 0; i < TPW; ++i) {
            const int t = warp + (SCAN_THREADS / 32) * i;
            if (t >= tc) continue;
            const float* row = qkv + (size_t)(start + t0 + t) * ldq;
            const float* abr = ab + (size_t)(start + t0 + t) * ldab;
            const float* alr = al + (size_t)(start + t0 + t) * ldal;
#pragma unroll
            for (int n = 0; n < NQ; ++n) {
                const int c4 = lane + 32 * n;
                pq[i][n] = make_float4(0.f, 0.f, 0.f, 0.f);
                pk[i][n] = pq[i][n];
                if (c4 < DP / 4 && c4 * 4 < d) {
                    pq[i][n] = *reinterpret_cast<const float4*>(row + q_off + kh * d + c4 * 4);
                    pk[i][n] = *reinterpret_cast<const float4*>(row + k_off + kh * d + c4 * 4);
                }
            }
            pv[i] = v0 + lane < dv ? row[v_off + h * dv + v0 + lane] : 0.f;
            if (CH) {
#pragma unroll
                for (int n = 0; n < NA; ++n) {
                    const int c = lane + 32 * n;
                    pa[i][n] = c < d ? alr[a_off + h * d + c] : 0.f;
                }
            } else {
                pa[i][0] = lane == 0 ? alr[a_off + h] : 0.f;
            }
            pb[i] = lane == 0 ? abr[b_off + h] : 0.f;
        }
    };
    if (vec) fetch(0);
    for (int t0 = 0; t0 < len; t0 += TC) {
        const int tc = min(TC, len - t0);
        __syncthreads();
        // raw q, k and v of a warp's tokens into shared memory, then q and k as unit vectors (sum of squares: a
        // lane's elements in order, then a tree over the lanes)
        float sq[TPW], sk[TPW];
#pragma unroll
        for (int i = 0; i < TPW; ++i) {
            const int t = warp + (SCAN_THREADS / 32) * i;
            sq[i] = 0.f; sk[i] = 0.f;
            if (t >= tc) continue;
            const float* row = qkv + (size_t)(start + t0 + t) * ldq;
            const float* abr = ab + (size_t)(start + t0 + t) * ldab;
            const float* alr = al + (size_t)(start + t0 + t) * ldal;
            if (vec) {
#pragma unroll
                for (int n = 0; n < NQ; ++n) {
                    const int c4 = lane + 32 * n;
                    if (c4 >= DP / 4) continue;
                    const float4 qv = pq[i][n], kv = pk[i][n];
                    *reinterpret_cast<float4*>(&q_s[t][c4 * 4]) = qv;
                    *reinterpret_cast<float4*>(&k_s[t][c4 * 4]) = kv;
                    sq[i] = fmaf(qv.x, qv.x, sq[i]); sq[i] = fmaf(qv.y, qv.y, sq[i]);
                    sq[i] = fmaf(qv.z, qv.z, sq[i]); sq[i] = fmaf(qv.w, qv.w, sq[i]);
                    sk[i] = fmaf(kv.x, kv.x, sk[i]); sk[i] = fmaf(kv.y, kv.y, sk[i]);
                    sk[i] = fmaf(kv.z, kv.z, sk[i]); sk[i] = fmaf(kv.w, kv.w, sk[i]);
                }
                v_s[t][lane] = pv[i];
                if (CH) {
#pragma unroll
                    for (int n = 0; n < NA; ++n) {
                        const int c = lane + 32 * n;
                        if (c < DP) gc_s[t][c] = c < d ? expf(-rate * rc_softplus(pa[i][n] + dtc[n])) : 1.f;
                    }
                }
                if (lane == 0) {
                    if (!CH) g_s[t] = expf(-rate * rc_softplus(pa[i][0] + dt));
                    b_s[t] = rc_sigmoid(pb[i]);
                }
                continue;
            }
            for (int c = lane; c < DP; c += 32) {
                const float qv = c < d ? row[q_off + kh * d + c] : 0.f;
                const float kv = c < d ? row[k_off + kh * d + c] : 0.f;
                q_s[t][c] = qv; k_s[t][c] = kv;
                sq[i] = fmaf(qv, qv, sq[i]); sk[i] = fmaf(kv, kv, sk[i]);
            }
            v_s[t][lane] = v0 + lane < dv ? row[v_off + h * dv + v0 + lane] : 0.f;
            if (CH) {
                for (int c = lane; c < DP; c += 32)
                    gc_s[t][c] = c < d ? expf(-rate * rc_softplus(alr[a_off + h * d + c] + load_w(dt_bias, p_dtype, h * d + c))) : 1.f;
            }
            if (lane == 0) {
                if (!CH) g_s[t] = expf(-rate * rc_softplus(alr[a_off + h] + dt));
                b_s[t] = rc_sigmoid(abr[b_off + h]);
            }
        }
#pragma unroll
        for (int i = 0; i < TPW; ++i) {
            const int t = warp + (SCAN_THREADS / 32) * i;
            if (t >= tc) continue;
            const float iq = q_scale / sqrtf(warp_sum(sq[i]) + unit_eps), ik = 1.f / sqrtf(warp_sum(sk[i]) + unit_eps);
            for (int c = lane; c < DP; c += 32) { q_s[t][c] *= iq; k_s[t][c] *= ik; }
        }
        __syncthreads();
        if (vec && t0 + TC < len) fetch(t0 + TC);
        for (int t = 0; t < tc; ++t) {
            const float g = CH ? 1.f : g_s[t];
            float r0 = 0.f, r1 = 0.f, r2 = 0.f, r3 = 0.f;     // four chains instead of one of R dependent steps
#pragma unroll
            for (int i = 0; i < R / 4; ++i) {
                const float4 kk = *reinterpret_cast<const float4*>(&k_s[t][KEY_OF(i, part)]);
                float4 gg = make_float4(g, g, g, g);
                if (CH) gg = *reinterpret_cast<const float4*>(&gc_s[t][KEY_OF(i, part)]);
                S[4 * i] *= gg.x;      r0 = fmaf(S[4 * i], kk.x, r0);
                S[4 * i + 1] *= gg.y;  r1 = fmaf(S[4 * i + 1], kk.y, r1);
                S[4 * i + 2] *= gg.z;  r2 = fmaf(S[4 * i + 2], kk.z, r2);
                S[4 * i + 3] *= gg.w;  r3 = fmaf(S[4 * i + 3], kk.w, r3);
            }
            const float r = part_sum<P>((r0 + r1) + (r2 + r3));
            const float u = b_s[t] * (v_s[t][vl] - r);
            float o0 = 0.f, o1 = 0.f, o2 = 0.f, o3 = 0.f;
#pragma unroll
            for (int i = 0; i < R / 4; ++i) {
                const float4 kk = *reinterpret_cast<const float4*>(&k_s[t][KEY_OF(i, part)]);
                const float4 qq = *reinterpret_cast<const float4*>(&q_s[t][KEY_OF(i, part)]);
                S[4 * i] = fmaf(kk.x, u, S[4 * i]);          o0 = fmaf(S[4 * i], qq.x, o0);
                S[4 * i + 1] = fmaf(kk.y, u, S[4 * i + 1]);  o1 = fmaf(S[4 * i + 1], qq.y, o1);
                S[4 * i + 2] = fmaf(kk.z, u, S[4 * i + 2]);  o2 = fmaf(S[4 * i + 2], qq.z, o2);
                S[4 * i + 3] = fmaf(kk.w, u, S[4 * i + 3]);  o3 = fmaf(S[4 * i + 3], qq.w, o3);
            }
            const float o = part_sum<P>((o0 + o1) + (o2 + o3));
            if (part == 0) o_s[t][vl] = o;
        }
        __syncthreads();
        for (int i = threadIdx.x; i < tc * SCAN_VS; i += SCAN_THREADS) {
            const int t = i / SCAN_VS, c = i - t * SCAN_VS;
            if (v0 + c < dv) out[(size_t)(start + t0 + t) * H * dv + h * dv + v0 + c] = o_s[t][c];
        }
    }
    if (live) scan_store_state<R, P>(S, st, part);
}

// ---- the gated delta rule over prompts
// The same recurrence in two kernels.  The first makes what a token needs once for all slices of value columns: q and k as
// unit vectors, the decays and beta (in the kernel above every block makes them again, 128 softpluses and exponentials a
// token, and a chunk's walk waits for its staging).  The second walks, a ring of asynchronous copies ahead, 8 tokens to a
// group; the read-outs of a group meet in one exchange.  Sums, products and their order are the kernel's above, and so are
// the bits.  What bounds it is the chain from one token's state to the next (decay, a sum of four, three exchanges, the
// write) in a scheduler that has one warp.
// Measured, 2,048 tokens, 16 heads of 128 x 128 on 8 key heads, a decay per channel: 1,015 us in one kernel, 374 us in two
// (the first 18).
#define DS_GROUP 8           // tokens to a group of the ring, the lanes of a column
#define DS_STAGES 4
#define DS_COLS 16           // value columns to a block

// qk [n, Hk, 2, d]: q (unit, times q_scale) and k (unit).  gb [n, H, d + 4] (CH) or [n, H, 4]: decays, then beta.  A warp per
// (token, key head) and per (token, head).
template <int CH>
__global__ void __launch_bounds__(256)
delta_prepare_kernel(const float* __restrict__ qkv, long long ldq, int q_off, int k_off, const float* __restrict__ ab,
                     long long ldab, int b_off, int a_off, const float* __restrict__ al, long long ldal,
                     const void* __restrict__ A_log, const void* __restrict__ dt_bias, int p_dtype, float* __restrict__ qk,
                     float* __restrict__ gb, long long n_items, int H, int Hk, int d, float unit_eps, float q_scale) {
    gi_pdl_start();
    const long long item = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (item >= n_items) return;
    const int lane = threadIdx.x & 31, c = lane * 4;
    const long long t = item / (H + Hk);
    const int part = (int)(item - t * (H + Hk));
    if (part < Hk) {
        const float* row = qkv + t * ldq + (size_t)part * d;
        float4 q = make_float4(0.f, 0.f, 0.f, 0.f), k = q;
        float sq = 0.f, sk = 0.f;
        if (c < d) {
            q = *reinterpret_cast<const float4*>(row + q_off + c);
            k = *reinterpret_cast<const float4*>(row + k_off + c);
        }
        sq = fmaf(q.x, q.x, sq); sq = fmaf(q.y, q.y, sq); sq = fmaf(q.z, q.z, sq); sq = fmaf(q.w, q.w, sq);
        sk = fmaf(k.x, k.x, sk); sk = fmaf(k.y, k.y, sk); sk = fmaf(k.z, k.z, sk); sk = fmaf(k.w, k.w, sk);
        const float iq = q_scale / sqrtf(warp_sum(sq) + unit_eps), ik = 1.f / sqrtf(warp_sum(sk) + unit_eps);
        if (c < d) {
            float* dst = qk + (t * Hk + part) * (2LL * d) + c;
            *reinterpret_cast<float4*>(dst) = make_float4(q.x * iq, q.y * iq, q.z * iq, q.w * iq);
            *reinterpret_cast<float4*>(dst + d) = make_float4(k.x * ik, k.y * ik, k.z * ik, k.w * ik);
        }
        return;
    }
    const int h = part - Hk;
    const float rate = expf(load_w(A_log, p_dtype, h));
    const float* a = al + t * ldal + a_off;
    float* dst = gb + (t * H + h) * (CH ? d + 4LL : 4LL);
    if (CH && c < d) {
        float4 g;
        g.x = expf(-rate * rc_softplus(a[h * d + c] + load_w(dt_bias, p_dtype, h * d + c)));
        g.y = expf(-rate * rc_softplus(a[h * d + c + 1] + load_w(dt_bias, p_dtype, h * d + c + 1)));
        g.z = expf(-rate * rc_softplus(a[h * d + c + 2] + load_w(dt_bias, p_dtype, h * d + c + 2)));
        g.w = expf(-rate * rc_softplus(a[h * d + c + 3] + load_w(dt_bias, p_dtype, h * d + c + 3)));
        *reinterpret_cast<float4*>(dst + c) = g;
    }
    if (lane == 0) {
        const float g = CH ? 0.f : expf(-rate * rc_softplus(a[h] + load_w(dt_bias, p_dtype, h)));
        *reinterpret_cast<float4*>(dst + (CH ? d : 0)) = make_float4(rc_sigmoid(ab[t * ldab + b_off + h]), g, 0.f, 0.f);
    }
}

// Keys of D = 8 R, W value columns to a thread.  spans [n_seq, 3]; out float32 [n, H dv].  qk and gb hold rows row0 .. row1 - 1
// of the step; the rows before were walked by earlier launches, whose state this one goes on from.
template <int R, int CH, int W>
__global__ void __launch_bounds__(DS_COLS / W * 8, 1)
delta_walk_kernel(const float* __restrict__ qk, const float* __restrict__ gb, const float* __restrict__ qkv, long long ldq, int v_off,
                  float* __restrict__ state, long long state_stride, const int* __restrict__ spans, float* __restrict__ out, int H,
                  int Hk, int dv, int row0, int row1) {
    gi_pdl_start();
    constexpr int P = 8, D = R * P, DS_THREADS = DS_COLS / W * P, GB = CH ? D + 4 : 4;       // floats of a row of decays and beta
    constexpr int TOKEN = 2 * D + GB + DS_COLS, QK_COPIES = 2 * D / 4, G_COPIES = CH ? D / 4 : 0;      // a token's floats, its 16-byte copies
    extern __shared__ __align__(16) float ds_smem[];                   // [stage][token][q | k | decays, beta | v]
    const int slot = spans[3 * blockIdx.x], start = max(spans[3 * blockIdx.x + 1], row0);
    const int len = min(spans[3 * blockIdx.x + 1] + spans[3 * blockIdx.x + 2], row1) - start;      // the span's rows of this launch
    if (len <= 0) return;
    const int h = blockIdx.y, v0 = blockIdx.z * DS_COLS, kh = h / (H / Hk), tid = threadIdx.x;
    const int part = tid % P, col = tid / P * W;                       // this thread's columns: v0 + col (and the next)
    if (slot < 0) {
        for (int t = 0; t < len; ++t)
            if (part < W) out[(size_t)(start + t) * H * dv + h * dv + v0 + col + part] = 0.f;
        return;
    }
    const int groups = (len + DS_GROUP - 1) / DS_GROUP;
    const uint32_t smem0 = (uint32_t)__cvta_generic_to_shared(ds_smem);
    auto copy = [&](uint32_t dst, const float* src) { asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(src)); };
    // a group's tokens beyond the sequence's end are its last token again, and not walked
    auto fetch = [&](int grp) {
        if (grp < groups) {
            const uint32_t base = smem0 + (uint32_t)(grp % DS_STAGES) * (DS_GROUP * TOKEN * 4);
            const int t0 = grp * DS_GROUP, last = len - 1;
#pragma unroll
            for (int i = 0; i < DS_GROUP * QK_COPIES / DS_THREADS; ++i) {
                const int id = tid + DS_THREADS * i, j = id / QK_COPIES, c = id % QK_COPIES;
                copy(base + (j * TOKEN + 4 * c) * 4, qk + ((size_t)(start - row0 + min(t0 + j, last)) * Hk + kh) * (2 * D) + 4 * c);
            }
#pragma unroll
            for (int i = 0; i < DS_GROUP * G_COPIES / DS_THREADS; ++i) {
                const int id = tid + DS_THREADS * i, j = id / (G_COPIES ? G_COPIES : 1), c = id % (G_COPIES ? G_COPIES : 1);
                copy(base + (j * TOKEN + 2 * D + 4 * c) * 4, gb + ((size_t)(start - row0 + min(t0 + j, last)) * H + h) * GB + 4 * c);
            }
            if (tid < 32) {
                const int j = tid / 4, c = tid % 4;
                copy(base + (j * TOKEN + 2 * D + GB + 4 * c) * 4, qkv + (size_t)(start + min(t0 + j, last)) * ldq + v_off + h * dv + v0 + 4 * c);
            } else if (tid < 40) {
                const int j = tid - 32;
                copy(base + (j * TOKEN + 2 * D + GB - 4) * 4, gb + ((size_t)(start - row0 + min(t0 + j, last)) * H + h) * GB + GB - 4);
            }
        }
        asm volatile("cp.async.commit_group;\n" ::);
    };
    for (int g = 0; g < DS_STAGES - 1; ++g) fetch(g);
    float* st = state + (size_t)slot * state_stride + ((size_t)h * dv + v0 + col) * D;
    f32x2 S[W][R / 2];
#pragma unroll
    for (int w = 0; w < W; ++w) scan_load_pairs<R, P>(S[w], st + w * D, part, true);
    float* dst = out + (size_t)start * H * dv + h * dv + v0 + col;
    for (int grp = 0; grp < groups; ++grp) {
        asm volatile("cp.async.wait_group %0;\n" ::"n"(DS_STAGES - 2));
        __syncthreads();                                               // the group is there, and the one before it is done with
        fetch(grp + DS_STAGES - 1);
        const int left = len - grp * DS_GROUP;
        float o[W][P];
        // Token j: its operands come out of shared memory while the token before is walked, and what is read of the state
        // with that token's q is summed beside the decay and the sum with this one's k, so that neither lies in the chain.
        struct Operands { f32x2 k[R / 2], g[CH ? R / 2 : 1], q[R / 2]; float beta, v[W]; };
        // (volatile, so that they stay ahead of the exchanges of the token that is walked)
        const uint32_t tok_addr = smem0 + (uint32_t)(grp % DS_STAGES) * (DS_GROUP * TOKEN * 4);
        auto pair = [](uint32_t at, f32x2& x, f32x2& y) { asm volatile("ld.shared.v2.u64 {%0, %1}, [%2];" : "=l"(x), "=l"(y) : "r"(at)); };
        auto operands = [&](Operands& a, int j) {
            const uint32_t x = tok_addr + j * (TOKEN * 4);
#pragma unroll
            for (int i = 0; i < R / 4; ++i) {
                pair(x + (D + KEY_OF(i, part)) * 4, a.k[2 * i], a.k[2 * i + 1]);
                if (CH) pair(x + (2 * D + KEY_OF(i, part)) * 4, a.g[CH ? 2 * i : 0], a.g[CH ? 2 * i + 1 : 0]);
            }
            float decay;                                               // of the whole head
            asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(a.beta), "=f"(decay) : "r"(x + (2 * D + GB - 4) * 4));
            if (!CH) a.g[0] = both2(decay);
#pragma unroll
            for (int w = 0; w < W; ++w) asm volatile("ld.shared.f32 %0, [%1];" : "=f"(a.v[w]) : "r"(x + (2 * D + GB + col + w) * 4));
#pragma unroll
            for (int i = 0; i < R / 4; ++i) pair(x + KEY_OF(i, part) * 4, a.q[2 * i], a.q[2 * i + 1]);
        };
        auto read = [&](const Operands& a, int j) {
#pragma unroll
            for (int w = 0; w < W; ++w) {
                f32x2 oa = 0ull, ob = 0ull;
#pragma unroll
                for (int i = 0; i < R / 4; ++i) {
                    oa = fma2(S[w][2 * i], a.q[2 * i], oa);
                    ob = fma2(S[w][2 * i + 1], a.q[2 * i + 1], ob);
                }
                o[w][j] = sum2(oa, ob);
            }
        };
        auto write = [&](const Operands& a) {
            f32x2 ra[W], rb[W];
#pragma unroll
            for (int w = 0; w < W; ++w) {
                ra[w] = rb[w] = 0ull;
#pragma unroll
                for (int i = 0; i < R / 4; ++i) {
                    S[w][2 * i] = mul2(S[w][2 * i], a.g[CH ? 2 * i : 0]);
                    S[w][2 * i + 1] = mul2(S[w][2 * i + 1], a.g[CH ? 2 * i + 1 : 0]);
                    ra[w] = fma2(S[w][2 * i], a.k[2 * i], ra[w]);
                    rb[w] = fma2(S[w][2 * i + 1], a.k[2 * i + 1], rb[w]);
                }
            }
            float r[W];
#pragma unroll
            for (int w = 0; w < W; ++w) r[w] = sum2(ra[w], rb[w]);
#pragma unroll
            for (int off = 1; off < P; off <<= 1)                      // part_sum of every column, side by side
#pragma unroll
                for (int w = 0; w < W; ++w) r[w] += __shfl_xor_sync(0xffffffffu, r[w], off);
#pragma unroll
            for (int w = 0; w < W; ++w) {
                const f32x2 u = both2(a.beta * (a.v[w] - r[w]));
#pragma unroll
                for (int i = 0; i < R / 2; ++i) S[w][i] = fma2(a.k[i], u, S[w][i]);
            }
        };
        Operands a[2];
        if (left >= DS_GROUP) {                                        // no branch between tokens
            operands(a[0], 0);
#pragma unroll
            for (int j = 0; j < DS_GROUP; ++j) {
                if (j) read(a[(j + 1) & 1], j - 1);
                if (j + 1 < DS_GROUP) operands(a[(j + 1) & 1], j + 1);
                write(a[j & 1]);
            }
            read(a[(DS_GROUP - 1) & 1], DS_GROUP - 1);
        } else {
#pragma unroll
            for (int j = 0; j < DS_GROUP; ++j) {
#pragma unroll
                for (int w = 0; w < W; ++w) o[w][j] = 0.f;
                if (j < left) {                                        // the same for the whole block
                    operands(a[0], j);
                    write(a[0]);
                    read(a[0], j);
                }
            }
        }
        // token `part` of the group ends in lane `part`
        float y[W];
#pragma unroll
        for (int w = 0; w < W; ++w) y[w] = part_sum_tokens<P>(o[w], part);
        if (part < left) {
            float* at = dst + (size_t)(grp * DS_GROUP + part) * H * dv;
            if (W == 2) *reinterpret_cast<float2*>(at) = make_float2(y[0], y[W - 1]);
            else *at = y[0];
        }
    }
    asm volatile("cp.async.wait_group 0;\n" ::);
#pragma unroll
    for (int w = 0; w < W; ++w) scan_store_pairs<R, P>(S[w], st + w * D, part);
}

// Floats of one head's state for key dimension d and value dimension dv, as the scans lay it out.
extern "C" long long gi_scan_state_floats(int d, int dv) {
    const int dp = scan_padded(d);
    return dp ? (long long)dv * dp : -1;
}

extern "C" int gi_decay_scan(const void* qkv, long long ld, int act_dtype, int q_off, int k_off, int v_off,
                             const float* decay, float* state, long long state_stride, const int* spans,
                             const int* tok_slot, float* out, int n_seq, int H, int d, int dv, void* stream) {
    const int DP = scan_padded(d);
    GI_REQUIRE(n_seq >= 0 && H > 0 && d > 0 && dv > 0 && DP > 0, "gi_decay_scan: key dimension %d (at most 256)", d);
    GI_REQUIRE(H <= 65535 && (dv + SCAN_VS - 1) / SCAN_VS <= 65535, "gi_decay_scan: %d heads of %d values", H, dv);
    GI_REQUIRE(state_stride >= (long long)H * dv * DP && state_stride % 4 == 0, "gi_decay_scan: state rows of %lld "
               "floats are shorter than %lld or no multiple of 4", state_stride, (long long)H * dv * DP);
    if (n_seq == 0) return 0;
    cudaStream_t s = (cudaStream_t)stream;
    dim3 grid(n_seq, H, (dv + SCAN_VS - 1) / SCAN_VS);
    if (act_dtype == GI_DTYPE_F32) {
        SCAN_DISPATCH(decay_scan_kernel, float, (const float*)qkv, ld, q_off, k_off, v_off, decay, state, state_stride, spans, tok_slot, out, H, d, dv, 0)
    } else if (act_dtype == GI_DTYPE_BF16) {
        const int vec_rows = d % 8 == 0 && dv % 8 == 0 && ld % 8 == 0 && q_off % 8 == 0 && k_off % 8 == 0 && v_off % 8 == 0 &&
                             (uintptr_t)qkv % 16 == 0;
        SCAN_DISPATCH(decay_scan_kernel, bf16, (const bf16*)qkv, ld, q_off, k_off, v_off, decay, state, state_stride, spans, tok_slot, out, H, d, dv, vec_rows)
    } else {
        GI_REQUIRE(false, "gi_decay_scan: activation dtype %d", act_dtype);
    }
    return gi_check_launch("gi_decay_scan");
}

extern "C" int gi_delta_scan(const float* qkv, long long ldq, int q_off, int k_off, int v_off, const float* ab,
                             long long ldab, int b_off, int a_off, const float* a_sep, long long lda_sep,
                             const void* A_log, const void* dt_bias,
                             int p_dtype, float* state, long long state_stride, const int* spans, const int* tok_slot,
                             float* out, int n_seq, int H, int Hk, int d, int dv, float unit_eps, float q_scale,
                             int channel_decay, void* stream) {
    const int DP = scan_padded(d);
    GI_REQUIRE(n_seq >= 0 && H > 0 && Hk > 0 && H % Hk == 0 && d > 0 && dv > 0 && DP > 0,
               "gi_delta_scan: %d heads on %d key heads, key dimension %d (at most 256)", H, Hk, d);
    GI_REQUIRE(H <= 65535 && (dv + SCAN_VS - 1) / SCAN_VS <= 65535, "gi_delta_scan: %d heads of %d values", H, dv);
    GI_REQUIRE(state_stride >= (long long)H * dv * DP && state_stride % 4 == 0, "gi_delta_scan: state rows of %lld "
               "floats are shorter than %lld or no multiple of 4", state_stride, (long long)H * dv * DP);
    if (n_seq == 0) return 0;
    cudaStream_t s = (cudaStream_t)stream;
    dim3 grid(n_seq, H, (dv + SCAN_VS - 1) / SCAN_VS);
    const int vec = d % 4 == 0 && ldq % 4 == 0 && q_off % 4 == 0 && k_off % 4 == 0 && (uintptr_t)qkv % 16 == 0;
    // the decay's logits: columns of `ab`, or a matrix of their own
    const float* al = a_sep ? a_sep : ab;
    const long long ldal = a_sep ? lda_sep : ldab;
    if (channel_decay) {
        SCAN_DISPATCH_X(delta_scan_kernel, float, SCAN_COMMA(1), qkv, ldq, q_off, k_off, v_off, ab, ldab, b_off, a_off, al, ldal, A_log, dt_bias, p_dtype, state, state_stride, spans, tok_slot, out, H, Hk, d, dv, unit_eps, q_scale, vec)
    } else {
        SCAN_DISPATCH_X(delta_scan_kernel, float, SCAN_COMMA(0), qkv, ldq, q_off, k_off, v_off, ab, ldab, b_off, a_off, al, ldal, A_log, dt_bias, p_dtype, state, state_stride, spans, tok_slot, out, H, Hk, d, dv, unit_eps, q_scale, vec)
    }
    return gi_check_launch("gi_delta_scan");
}

// gi_delta_scan over prompts by the two kernels above: keys of 64 or 128, values in whole blocks of columns, rows of qkv and of
// the state that start on 16 bytes.  `scratch`: scratch_rows (2 Hk d + H (d + 4 or 4)) floats, on 16 bytes; a step of more rows is
// walked that many at a time, each from the state that the one before left.
extern "C" int gi_delta_scan_prompt(const float* qkv, long long ldq, int q_off, int k_off, int v_off, const float* ab,
                                    long long ldab, int b_off, int a_off, const float* a_sep, long long lda_sep,
                                    const void* A_log, const void* dt_bias, int p_dtype, float* state, long long state_stride,
                                    const int* spans, float* out, float* scratch, int scratch_rows, int n_rows, int n_seq, int H, int Hk, int d,
                                    int dv, float unit_eps, float q_scale, int channel_decay, void* stream) {
    GI_REQUIRE(n_seq >= 0 && n_rows >= 0 && H > 0 && Hk > 0 && H % Hk == 0 && (d == 64 || d == 128) && dv > 0 && dv % DS_COLS == 0,
               "gi_delta_scan_prompt: %d heads on %d key heads, keys of %d, values of %d", H, Hk, d, dv);
    GI_REQUIRE(H <= 65535 && dv / DS_COLS <= 65535, "gi_delta_scan_prompt: %d heads of %d values", H, dv);
    GI_REQUIRE(state_stride >= (long long)H * dv * d && state_stride % 4 == 0 && (uintptr_t)state % 16 == 0,
               "gi_delta_scan_prompt: state rows of %lld floats", state_stride);
    GI_REQUIRE(ldq % 4 == 0 && q_off % 4 == 0 && k_off % 4 == 0 && v_off % 4 == 0 && ((uintptr_t)qkv | (uintptr_t)scratch) % 16 == 0 &&
               (uintptr_t)out % 8 == 0, "gi_delta_scan_prompt: rows start on 16 bytes");
    if (n_seq == 0 || n_rows == 0) return 0;
    cudaStream_t s = (cudaStream_t)stream;
    const float* al = a_sep ? a_sep : ab;
    const long long ldal = a_sep ? lda_sep : ldab;
    GI_REQUIRE(scratch_rows > 0, "gi_delta_scan_prompt: room for %d rows", scratch_rows);
    if (scratch_rows > n_rows) scratch_rows = n_rows;
    float *qk = scratch, *gb = scratch + (size_t)scratch_rows * Hk * 2 * d;
    GI_REQUIRE(((long long)scratch_rows * (H + Hk) + 7) / 8 <= 0x7fffffff, "gi_delta_scan_prompt: %d rows", scratch_rows);
    const auto prepare = channel_decay ? delta_prepare_kernel<1> : delta_prepare_kernel<0>;
    const size_t smem = (size_t)DS_STAGES * DS_GROUP * (2 * d + (channel_decay ? d + 4 : 4) + DS_COLS) * sizeof(float);
    // One column to a thread where the blocks fit the SMs side by side: four warps to an SM, one to a scheduler.  Two columns
    // beyond: half the reads of shared memory, which then are what several blocks to an SM wait for.
    const bool few = (long long)n_seq * H * (dv / DS_COLS) <= 148;
#define DS_WALK(R, CH) (few ? delta_walk_kernel<R, CH, 1> : delta_walk_kernel<R, CH, 2>)
    const auto walk = d == 128 ? (channel_decay ? DS_WALK(16, 1) : DS_WALK(16, 0)) : (channel_decay ? DS_WALK(8, 1) : DS_WALK(8, 0));
#undef DS_WALK
    if (int rc = gi_reserve_smem((const void*)walk, smem, "gi_delta_scan_prompt")) return rc;
    for (long long row0 = 0; row0 < n_rows; row0 += scratch_rows) {
        const int rows = (int)(n_rows - row0 < scratch_rows ? n_rows - row0 : scratch_rows);
        const long long items = (long long)rows * (H + Hk);
        gi_launch(prepare, dim3((unsigned)((items + 7) / 8)), dim3(256), 0, s, qkv + row0 * ldq, ldq, q_off, k_off, ab + row0 * ldab, ldab,
                  b_off, a_off, al + row0 * ldal, ldal, A_log, dt_bias, p_dtype, qk, gb, items, H, Hk, d, unit_eps, q_scale);
        if (int rc = gi_check_launch("gi_delta_scan_prompt")) return rc;
        gi_launch(walk, dim3(n_seq, H, dv / DS_COLS), dim3(few ? DS_COLS * 8 : DS_COLS * 4), smem, s, (const float*)qk, (const float*)gb, qkv,
                  ldq, v_off, state, state_stride, spans, out, H, Hk, dv, (int)row0, (int)row0 + rows);
        if (int rc = gi_check_launch("gi_delta_scan_prompt")) return rc;
    }
    return 0;
}
