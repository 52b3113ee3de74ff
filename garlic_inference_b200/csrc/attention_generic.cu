// Attention over the paged cache for any number of new tokens per sequence,
// float32 or bfloat16, any head_dim up to 1024.
//
// This is the engine's exact path: the float32 engine uses it for prompts and
// for decoding alike, and the bfloat16 engine uses it for head sizes its
// tensor-core kernels do not take.  One block computes one (token, query
// head).  Keys are visited in chunks of 32 aligned to absolute positions
// (chunk c = keys 32c..32c+31), chunk c by warp c mod 4, and the four partial
// results are merged in warp order: the result at a position therefore does
// not depend on how the tokens were cut into steps, on the batch, or on where
// the pages lie.
//
//   o = softmax_j( q . k_j * scale ) v_j   over keys j <= pos, and j > pos - window
//                                           when window > 0
// With `sinks` (one number per query head) the softmax's denominator also holds exp(sink_h): a key without a
// value, not scaled, counted once.  With d_v < d only the first d_v columns of a value row are summed and the
// output rows are d_v wide (a cache whose rows serve as keys in full and as values in part).
// Query head h reads key/value head h / (n_q / n_kv).  Scores, softmax and the
// weighted sum are float32.
// Three more parameters, for mixers beside plain grouped-query attention:
//   chunk > 0    a query at position i sees only the keys j <= i of its own chunk, floor(j / chunk) = floor(i / chunk)
//                (chunks are counted from position 0 of the sequence);
//   values of their own shape: the value pool has n_vh heads per page with rows of v_row elements, which may be
//                wider or narrower than a key row;
//   maps > 1     every head owns `maps` softmaxes over the same values (the maps of a differential attention):
//                the n_q query rows of a token are laid out [head][map], the n_kv key heads [key head][map], and
//                row h = head * maps + map reads key head (head / group) * maps + map and value head head / group,
//                group = (n_q / maps) / n_vh;
//   dist_bias    a learned bias per distance and query row, float32 [n_dist, n_q]: the score of key j for the query at
//                position i gets dist_bias[min(i - j, n_dist - 1), row] added after the scaling;
//   means        beside the keys of its window a query sees one more row (key and value) for every block of `block`
//                positions that lies wholly before the window, block b from b block + block - 1 <= i - window on; they
//                come from pools of their own and share the softmax (a window is required then).  They are visited
//                before the window's keys, 32 at a time like those;
//   keep_first   the first `keep_first` positions of a sequence stay in sight of every later query beside the window (a
//                window is required); like block rows they are visited before the window's keys, 32 at a time;
//   out_f32      the result is written as float32 whatever the activation type is (a later kernel combines maps).  Upstream hands this to a library
// (src/src-cuda/attention/fattn.cu:74-86: scale 1/sqrt(head_dim), causal mask
// aligned to the last key, float32 intermediates).
#include "common.cuh"
#include <math.h>
#include <type_traits>

#define AG_WARPS 4
#define AR_BLOCKS 148        // blocks from which on rows share their fetches

// Rows that stand for whole blocks of positions: row b of a sequence in page b / rows of its row of `table`, at row
// b % rows; pools [pages, heads, rows, width].  block = 0: none.
struct BlockRows {
    const void *k, *v;
    const int* table;
    int block, rows, max_pages, n_pages;
};

template <typename T> struct Vec;
template <> struct Vec<float> { static constexpr int N = 4; typedef float4 type; };
template <> struct Vec<bf16> { static constexpr int N = 8; typedef uint4 type; };

__device__ __forceinline__ float dot_vec(const float4& k, const float* q) {
    return k.x * q[0] + k.y * q[1] + k.z * q[2] + k.w * q[3];
}
__device__ __forceinline__ float dot_vec(const uint4& k, const float* q) {
    const __nv_bfloat162* k2 = reinterpret_cast<const __nv_bfloat162*>(&k);
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float2 f = __bfloat1622float2(k2[i]);
        s += f.x * q[2 * i] + f.y * q[2 * i + 1];
    }
    return s;
}

template <typename T, int DPL>
__global__ void __launch_bounds__(AG_WARPS * 32)
attn_generic_kernel(const T* __restrict__ q, const T* __restrict__ k_pool, const T* __restrict__ v_pool,
                    const int* __restrict__ block_table, const int* __restrict__ tok_pos,
                    const int* __restrict__ tok_slot, T* __restrict__ out, int n_q, int n_kv, int d,
                    int page_size, int max_pages, int n_pool_pages, int window, float scale,
                    const void* __restrict__ sinks, int sink_dtype, int d_v, int* __restrict__ status,
                    int chunk, int n_vh, int v_row, int maps, float* __restrict__ out_f32,
                    const float* __restrict__ dist_bias, int n_dist, BlockRows means, int keep_first) {
    gi_pdl_start();
    extern __shared__ float smem[];
    const int dw = d > d_v ? d : d_v;        // width of an accumulator row
    float* q_s = smem;                       // d
    float* acc_s = smem + d;                 // AG_WARPS * dw
    float* m_s = acc_s + AG_WARPS * dw;      // AG_WARPS
    float* l_s = m_s + AG_WARPS;             // AG_WARPS

    const int t = blockIdx.x, h = blockIdx.y;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    T* o = out ? out + ((size_t)t * n_q + h) * d_v : nullptr;
    float* of = out_f32 ? out_f32 + ((size_t)t * n_q + h) * d_v : nullptr;
    const int slot = tok_slot[t];
    const int pos = tok_pos[t];
    if (slot < 0 || pos < 0 || pos / page_size >= max_pages) {
        for (int i = threadIdx.x; i < d_v; i += blockDim.x) {
            if (of) of[i] = 0.f; else o[i] = from_f32<T>(0.f);
        }
        if (slot >= 0 && threadIdx.x == 0) atomicExch(status, 4);
        return;
    }
    const int head = h / maps, group = (n_q / maps) / n_vh;
    const int kvh = (head / group) * maps + (h - head * maps);
    const int vh = head / group;
    const T* qrow = q + ((size_t)t * n_q + h) * d;
    for (int i = threadIdx.x; i < d; i += blockDim.x) q_s[i] = to_f32(qrow[i]) * scale;
    __syncthreads();

    int lo = window > 0 ? max(0, pos - window + 1) : 0;
    if (chunk > 0) lo = max(lo, pos / chunk * chunk);
    const int* bt = block_table + (size_t)slot * max_pages;
    float m = -INFINITY, l = 0.f;
    float acc[DPL];
#pragma unroll
    for (int r = 0; r < DPL; ++r) acc[r] = 0.f;

    constexpr int VN = Vec<T>::N;
    typedef typename Vec<T>::type vec_t;
    // blocks the query sees: b with (b + 1) block <= pos - window + 1
    const int n_blocks = means.block > 0 && pos >= window ? (pos - window + 1) / means.block : 0;
    // first tokens that stay in sight: those that the window has left behind
    const int n_kept = window > 0 ? min(keep_first, lo) : 0;
    const int lead_chunks = (max(n_blocks, n_kept) + 31) / 32, first_chunk = lo / 32;
    const int padded = (lead_chunks + AG_WARPS - 1) / AG_WARPS * AG_WARPS;
    const int* mbt = means.block > 0 ? means.table + (size_t)slot * means.max_pages : nullptr;
    // the chunks of blocks (or of kept first tokens), then the chunks of keys: chunk c to warp c mod 4, counted from the
    // first of each kind
    for (int cc = warp; cc < padded + pos / 32 - first_chunk + 1; cc += AG_WARPS) {
        const bool lead = cc < padded, of_blocks = lead && means.block > 0;
        const int c = lead ? cc : cc - padded + first_chunk;
        const int j = c * 32 + lane;
        const bool valid = lead ? j < max(n_blocks, n_kept) : j >= lo && j <= pos;
        long long row = -1;                  // element offset of this lane's key row (-1: none)
        long long vrow = 0;                  // and of its value row
        float s = -INFINITY;
        const T* kp = of_blocks ? (const T*)means.k : k_pool;
        const T* vp = of_blocks ? (const T*)means.v : v_pool;
        if (valid) {
            const int rows = of_blocks ? means.rows : page_size, lp = j / rows;
            const int page = of_blocks ? (lp < means.max_pages ? mbt[lp] : -1) : bt[lp];
            if (page < 0 || page >= (of_blocks ? means.n_pages : n_pool_pages)) {
                atomicExch(status, 5);
            } else {
                row = (((long long)page * n_kv + kvh) * rows + (j - lp * rows)) * d;
                vrow = (((long long)page * n_vh + vh) * rows + (j - lp * rows)) * v_row;
                float a = 0.f;
                if (d % VN == 0) {               // rows start on 16 bytes: vector loads
                    const vec_t* kr = reinterpret_cast<const vec_t*>(kp + row);
                    for (int i = 0; i < d / VN; ++i) a += dot_vec(kr[i], q_s + i * VN);
                } else {
                    for (int i = 0; i < d; ++i) a = fmaf(to_f32(kp[row + i]), q_s[i], a);
                }
                s = dist_bias ? a + dist_bias[(size_t)min(pos - j, n_dist - 1) * n_q + h] : a;
            }
        }
        const float cmax = warp_max(s);
        if (cmax == -INFINITY) continue;
        const float m_new = fmaxf(m, cmax);
        const float corr = expf(m - m_new);              // 0 when m is -inf
        const float p = row >= 0 ? expf(s - m_new) : 0.f;
        l = l * corr + warp_sum(p);
        m = m_new;
#pragma unroll
        for (int r = 0; r < DPL; ++r) acc[r] *= corr;
        for (int jj = 0; jj < 32; ++jj) {
            const float pj = __shfl_sync(0xffffffffu, p, jj);
            const long long rj = __shfl_sync(0xffffffffu, row, jj);
            const long long vj = __shfl_sync(0xffffffffu, vrow, jj);
            if (rj < 0) continue;
            const T* vr = vp + vj;
#pragma unroll
            for (int r = 0; r < DPL; ++r) {
                const int i = lane + 32 * r;
                if (i < d_v) acc[r] += pj * to_f32(vr[i]);
            }
        }
    }
    if (lane == 0) { m_s[warp] = m; l_s[warp] = l; }
#pragma unroll
    for (int r = 0; r < DPL; ++r) {
        const int i = lane + 32 * r;
        if (i < dw) acc_s[warp * dw + i] = acc[r];
    }
    __syncthreads();
    float M = -INFINITY;
    for (int w = 0; w < AG_WARPS; ++w) M = fmaxf(M, m_s[w]);
    const float sink = sinks ? load_w(sinks, sink_dtype, h) : -INFINITY;
    M = fmaxf(M, sink);
    float L = 0.f;
    for (int w = 0; w < AG_WARPS; ++w) L += (m_s[w] == -INFINITY ? 0.f : expf(m_s[w] - M) * l_s[w]);
    if (sinks) L += expf(sink - M);
    for (int i = threadIdx.x; i < d_v; i += blockDim.x) {
        float v = 0.f;
        for (int w = 0; w < AG_WARPS; ++w)
            if (m_s[w] != -INFINITY) v += expf(m_s[w] - M) * acc_s[w * dw + i];
        const float res = L > 0.f ? v / L : 0.f;
        if (of) of[i] = res; else o[i] = from_f32<T>(res);
    }
}

template <typename T>
static int launch_generic(const void* q, const void* k_pool, const void* v_pool, const int* block_table,
                          const int* tok_pos, const int* tok_slot, void* out, int n_tokens, int n_q, int n_kv,
                          int d, int page_size, int max_pages, int n_pool_pages, int window, float scale,
                          const void* sinks, int sink_dtype, int d_v, int* status, int chunk, int n_vh, int v_row,
                          int maps, float* out_f32, const float* dist_bias, int n_dist, const BlockRows& means,
                          int keep_first, cudaStream_t s) {
    dim3 grid(n_tokens, n_q);
    const int dw = d > d_v ? d : d_v;
    const size_t smem = ((size_t)d + (size_t)dw * AG_WARPS + 2 * AG_WARPS) * sizeof(float);
#define AG_LAUNCH(DPL)                                                                               \
    gi_launch(attn_generic_kernel<T, DPL>, grid, dim3(AG_WARPS * 32), smem, s,                                     \
        (const T*)q, (const T*)k_pool, (const T*)v_pool, block_table, tok_pos, tok_slot, (T*)out,     \
        n_q, n_kv, d, page_size, max_pages, n_pool_pages, window, scale, sinks, sink_dtype, d_v, status, \
        chunk, n_vh, v_row, maps, out_f32, dist_bias, n_dist, means, keep_first)
    if (dw <= 32) AG_LAUNCH(1);
    else if (dw <= 64) AG_LAUNCH(2);
    else if (dw <= 128) AG_LAUNCH(4);
    else if (dw <= 256) AG_LAUNCH(8);
    else if (dw <= 512) AG_LAUNCH(16);
    else AG_LAUNCH(32);
#undef AG_LAUNCH
    return gi_check_launch("gi_attention_generic");
}

// The same for prompts of the float32 engine (no window, no chunks, one map): a block takes HR query heads of one key head and TQ
// neighbouring tokens of a sequence, whose rows share every key and value that is fetched.  Where neighbouring tokens are of several sequences
// (a decode step, short portions) each of these has a block of its own: TQ blocks stand by, one for every token that may be a sequence's first,
// the first tokens' in front.  Chunks, warps, sums and their order are
// the kernel's above for every row, and so are the bits.
// Bound above by the fetches (a block read every key and value of its token for one head, a key's row to a lane); here by the
// multiply-adds and the operands' reads from shared memory.  Measured, sequences of 300 and 200 tokens, 16 heads of 128 on 4 key heads: 223 us a
// row to a block, 92 us so (109 where a block took its tokens' sequences in turn).
template <int DPL, int HR, int TQ>
__global__ void __launch_bounds__(AG_WARPS * 32)
attn_shared_rows_kernel(const float* __restrict__ q, const float* __restrict__ k_pool, const float* __restrict__ v_pool,
                        const int* __restrict__ block_table, const int* __restrict__ tok_pos, const int* __restrict__ tok_slot,
                        float* __restrict__ out, int n_tokens, int n_q, int n_kv, int d, int page_size, int max_pages, int n_pool_pages,
                        float scale, const void* __restrict__ sinks, int sink_dtype, int d_v, int* __restrict__ status, int v_row) {
    gi_pdl_start();
    constexpr int R = HR * TQ;
    extern __shared__ __align__(16) float ar_smem[];
    const int dw = d > d_v ? d : d_v;
    float* q_s = ar_smem;                                    // [R][d]
    float* acc_s = q_s + R * d;                              // [AG_WARPS][R][dw]
    float* p_s = acc_s + AG_WARPS * R * dw;                  // [AG_WARPS][R][32], on 16 bytes: R is a multiple of 4
    float* m_s = p_s + AG_WARPS * R * 32;                    // [AG_WARPS][R]
    float* l_s = m_s + AG_WARPS * R;                         // [AG_WARPS][R]
    long long* v_s = reinterpret_cast<long long*>(l_s + AG_WARPS * R);       // [AG_WARPS][32]
    // (a prompt's last tokens first: they see most)
    const int t0 = (gridDim.x - 1 - blockIdx.x) * TQ, first = t0 + blockIdx.z, h0 = blockIdx.y * HR, kvh = h0 / (n_q / n_kv);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (first >= n_tokens) return;
    auto known = [&](int t) { return tok_slot[t] >= 0 && tok_pos[t] >= 0 && tok_pos[t] / page_size < max_pages; };
    const int at = tok_slot[first];                          // the block's sequence
    if (!known(first)) {
        for (int j = threadIdx.x; j < HR * d_v; j += AG_WARPS * 32) out[((size_t)first * n_q + h0) * d_v + j] = 0.f;
        if (at >= 0 && threadIdx.x == 0) atomicExch(status, 4);
        return;
    }
    if (first > t0 && tok_slot[first - 1] == at && known(first - 1)) return;        // a block before this one has it
    // its tokens, and the last position that they see
    int pos[TQ], n_mine = 0, last = -1;
#pragma unroll
    for (int i = 0; i < TQ; ++i) {
        const int t = first + i;
        if (n_mine == i && t < min(t0 + TQ, n_tokens) && tok_slot[t] == at && known(t)) ++n_mine;
        pos[i] = i < n_mine ? tok_pos[t] : -1;
        last = max(last, pos[i]);
    }
    for (int i = threadIdx.x; i < n_mine * HR * d; i += AG_WARPS * 32) {
        const int r = i / d, t = first + r / HR;
        q_s[i] = t < n_tokens ? q[((size_t)t * n_q + h0 + r % HR) * d + i % d] * scale : 0.f;
    }
    __syncthreads();
    float m[R], l[R], acc[R][DPL];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        m[r] = -INFINITY; l[r] = 0.f;
#pragma unroll
        for (int e = 0; e < DPL; ++e) acc[r][e] = 0.f;
    }
    // the rows 0 .. ROWS - 1
    const int* bt = block_table + (size_t)at * max_pages;
    auto walk = [&](auto rows) {
        constexpr int ROWS = decltype(rows)::value;
        for (int c = warp; c <= last / 32; c += AG_WARPS) {
            const int j = c * 32 + lane;
            long long row = -1, vrow = -1;                   // element offsets of this lane's key and value rows
            if (j <= last) {
                const int lp = j / page_size, page = bt[lp];
                if (page < 0 || page >= n_pool_pages) atomicExch(status, 5);
                else {
                    row = (((long long)page * n_kv + kvh) * page_size + (j - lp * page_size)) * d;
                    vrow = (((long long)page * n_kv + kvh) * page_size + (j - lp * page_size)) * v_row;
                }
            }
            float a[ROWS];
#pragma unroll
            for (int r = 0; r < ROWS; ++r) a[r] = 0.f;
            if (row >= 0) {
                const float4* kr = reinterpret_cast<const float4*>(k_pool + row);
#pragma unroll 8
                for (int i = 0; i < d / 4; ++i) {
                    const float4 k = kr[i];
#pragma unroll
                    for (int r = 0; r < ROWS; ++r) {
                        const float4 x = *reinterpret_cast<const float4*>(q_s + r * d + 4 * i);
                        const float y[4] = {x.x, x.y, x.z, x.w};
                        a[r] += dot_vec(k, y);
                    }
                }
            }
            __syncwarp();                                    // the chunk before is done with
            v_s[warp * 32 + lane] = vrow;
            bool any[ROWS];
#pragma unroll
            for (int r = 0; r < ROWS; ++r) {
                const bool sees = row >= 0 && j <= pos[r / HR];
                const float s = sees ? a[r] : -INFINITY, cmax = warp_max(s);
                any[r] = cmax != -INFINITY;
                float p = 0.f;
                if (any[r]) {
                    const float m_new = fmaxf(m[r], cmax), corr = expf(m[r] - m_new);
                    p = sees ? expf(s - m_new) : 0.f;
                    l[r] = l[r] * corr + warp_sum(p);
                    m[r] = m_new;
#pragma unroll
                    for (int e = 0; e < DPL; ++e) acc[r][e] *= corr;
                }
                p_s[(warp * R + r) * 32 + lane] = p;
            }
            __syncwarp();
            // four values' rows at a time
            for (int j4 = 0; j4 < 32; j4 += 4) {
                float v[4][DPL];
                bool there[4];
#pragma unroll
                for (int jj = 0; jj < 4; ++jj) {
                    const long long vj = v_s[warp * 32 + j4 + jj];
                    there[jj] = vj >= 0;
#pragma unroll
                    for (int e = 0; e < DPL; ++e) v[jj][e] = there[jj] && lane + 32 * e < d_v ? v_pool[vj + lane + 32 * e] : 0.f;
                }
#pragma unroll
                for (int r = 0; r < ROWS; ++r) {
                    const float4 p4 = *reinterpret_cast<const float4*>(p_s + (warp * R + r) * 32 + j4);
                    const float p[4] = {p4.x, p4.y, p4.z, p4.w};
#pragma unroll
                    for (int jj = 0; jj < 4; ++jj)
                        // (a row that does not see this key leaves its sums as they are, whatever the value is)
                        if (any[r] && there[jj] && c * 32 + j4 + jj <= pos[r / HR])
#pragma unroll
                            for (int e = 0; e < DPL; ++e) acc[r][e] += p[jj] * v[jj][e];
                }
            }
        }
    };
    if (n_mine == 1) walk(std::integral_constant<int, HR>{});
    else if (TQ > 2 && n_mine == 2) walk(std::integral_constant<int, 2 * HR>{});
    else walk(std::integral_constant<int, R>{});
    if (lane == 0)
#pragma unroll
        for (int r = 0; r < R; ++r) { m_s[warp * R + r] = m[r]; l_s[warp * R + r] = l[r]; }
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
        for (int e = 0; e < DPL; ++e)
            if (lane + 32 * e < dw) acc_s[(warp * R + r) * dw + lane + 32 * e] = acc[r][e];
    __syncthreads();
    for (int i = threadIdx.x; i < n_mine * HR * d_v; i += AG_WARPS * 32) {
        const int r = i / d_v, c = i % d_v, t = r / HR;
        float M = -INFINITY;
        for (int w = 0; w < AG_WARPS; ++w) M = fmaxf(M, m_s[w * R + r]);
        const float sink = sinks ? load_w(sinks, sink_dtype, h0 + r % HR) : -INFINITY;
        M = fmaxf(M, sink);
        float L = 0.f, v = 0.f;
        for (int w = 0; w < AG_WARPS; ++w) L += (m_s[w * R + r] == -INFINITY ? 0.f : expf(m_s[w * R + r] - M) * l_s[w * R + r]);
        if (sinks) L += expf(sink - M);
        for (int w = 0; w < AG_WARPS; ++w)
            if (m_s[w * R + r] != -INFINITY) v += expf(m_s[w * R + r] - M) * acc_s[(w * R + r) * dw + c];
        out[((size_t)(first + t) * n_q + h0 + r % HR) * d_v + c] = L > 0.f ? v / L : 0.f;
    }
}

template <int DPL, int HR, int TQ>
static int launch_shared_rows(const float* q, const float* k_pool, const float* v_pool, const int* block_table, const int* tok_pos,
                              const int* tok_slot, float* out, int n_tokens, int n_q, int n_kv, int d, int page_size, int max_pages,
                              int n_pool_pages, float scale, const void* sinks, int sink_dtype, int d_v, int* status, int v_row, cudaStream_t s) {
    constexpr int R = HR * TQ;
    const int dw = d > d_v ? d : d_v;
    const size_t smem = ((size_t)R * d + (size_t)AG_WARPS * R * dw + (size_t)AG_WARPS * R * 34) * sizeof(float) + AG_WARPS * 32 * sizeof(long long);
    const auto kernel = attn_shared_rows_kernel<DPL, HR, TQ>;
    if (int rc = gi_reserve_smem((const void*)kernel, smem, "gi_attention_generic")) return rc;
    gi_launch(kernel, dim3((n_tokens + TQ - 1) / TQ, n_q / HR, TQ), dim3(AG_WARPS * 32), smem, s, q, k_pool, v_pool, block_table, tok_pos, tok_slot, out,
              n_tokens, n_q, n_kv, d, page_size, max_pages, n_pool_pages, scale, sinks, sink_dtype, d_v, status, v_row);
    return gi_check_launch("gi_attention_generic");
}

// The general entry point: everything the file's head lists.  `out` is written in the activation type unless
// `out_f32` is given.  single: every token is of a sequence of its own (a decode step), which only the choice of kernel heeds.  Key rows whose width is a multiple of 16 bytes are read with vector loads, others
// element by element; value rows may have any width.
extern "C" int gi_attention_masked(const void* q, const void* k_pool, const void* v_pool, int act_dtype,
                                   const int* block_table, const int* tok_pos, const int* tok_slot,
                                   void* out, int n_tokens, int n_q, int n_kv, int d, int page_size,
                                   int max_pages, int n_pool_pages, int window, float scale, const void* sinks,
                                   int sink_dtype, int d_v, int* status, int chunk, int n_vh, int v_row, int maps,
                                   float* out_f32, const float* dist_bias, int n_dist, const void* mean_k,
                                   const void* mean_v, const int* mean_table, int mean_block, int mean_rows,
                                   int mean_max_pages, int mean_pages, int keep_first, int single, void* stream) {
    GI_REQUIRE(keep_first >= 0 && (keep_first == 0 || (window > 0 && chunk == 0 && mean_block == 0)), "gi_attention_generic: "
               "kept first tokens come with a window, without chunks and rows for blocks");
    GI_REQUIRE(n_tokens >= 0 && n_q > 0 && n_kv > 0 && d > 0, "gi_attention_generic: sizes must be positive");
    GI_REQUIRE(!dist_bias || n_dist > 0, "gi_attention_generic: a distance bias of %d rows", n_dist);
    GI_REQUIRE(maps >= 1 && n_vh >= 1 && n_q % maps == 0 && n_kv == n_vh * maps && (n_q / maps) % n_vh == 0,
               "gi_attention_generic: %d query rows and %d key heads in %d maps over %d value heads", n_q, n_kv, maps, n_vh);
    GI_REQUIRE(d <= 1024, "gi_attention_generic: head_dim %d is beyond 1024", d);
    GI_REQUIRE((uintptr_t)k_pool % 16 == 0, "gi_attention_generic: the key pool must start on 16 bytes");
    GI_REQUIRE(n_q <= 65535, "gi_attention_generic: %d query heads is beyond 65535", n_q);
    GI_REQUIRE(d_v > 0 && d_v <= v_row && d_v <= 1024, "gi_attention_generic: %d value columns of rows of %d", d_v, v_row);
    GI_REQUIRE(page_size > 0 && max_pages > 0 && window >= 0 && chunk >= 0, "gi_attention_generic: page size, table width, window and chunk");
    GI_REQUIRE(out || out_f32, "gi_attention_generic: no output");
    GI_REQUIRE(mean_block == 0 || (mean_block > 0 && window > 0 && chunk == 0 && !dist_bias && mean_rows > 0 && mean_max_pages > 0 &&
               mean_pages > 0 && (uintptr_t)mean_k % 16 == 0), "gi_attention_generic: rows for blocks of %d positions come with a window, "
               "without chunks and distance biases", mean_block);
    const BlockRows means = {mean_k, mean_v, mean_table, mean_block, mean_rows, mean_max_pages, mean_pages};
    if (n_tokens == 0) return 0;
    cudaStream_t s = (cudaStream_t)stream;
    // Many tokens of plain heads in float32: rows that share their fetches, where that leaves a block for every SM.  In us, a block a row / so,
    // 16 heads of 128 on 4 key heads, new tokens behind cached ones: 32 behind none 15 / 21, 64 behind none 17 / 22, 64 behind 2,000 357 / 220, 128
    // behind none 44 / 28, 400 behind none 261 / 100; on 8 key heads 128 behind none 46 / 28; 32 heads of 64 on 8 100 behind none 39 / 19; 64 single
    // tokens of 32 heads of 128 on 8 behind 2,000 846 / 472, 60 and a portion of 300 behind 500 1,240 / 353.  Not where every token is of a
    // sequence of its own and so is every head (`single`, one query head a key head): nothing is shared then, and the registers leave fewer
    // warps to wait: 64 of 16 heads of 128 behind 300 104 / 123.
    const int group = n_q / n_kv, hr = group % 4 == 0 ? 4 : group % 2 == 0 ? 2 : 1, tq = hr == 4 ? 2 : 4;
    if (act_dtype == GI_DTYPE_F32 && !(single && hr == 1) && (long long)((n_tokens + tq - 1) / tq) * (n_q / hr) >= AR_BLOCKS && window == 0 && chunk == 0 && maps == 1 && out && !out_f32 && !dist_bias && mean_block == 0 &&
        n_vh == n_kv && d % 4 == 0 && d <= 128 && d_v <= 128 && (uintptr_t)q % 16 == 0) {
#define AR_LAUNCH(DPL, HR, TQ) return launch_shared_rows<DPL, HR, TQ>((const float*)q, (const float*)k_pool, (const float*)v_pool, block_table, tok_pos, \
            tok_slot, (float*)out, n_tokens, n_q, n_kv, d, page_size, max_pages, n_pool_pages, scale, sinks, sink_dtype, d_v, status, v_row, s)
        if (d <= 64 && d_v <= 64) {
            if (hr == 4) AR_LAUNCH(2, 4, 2);
            if (hr == 2) AR_LAUNCH(2, 2, 4);
            AR_LAUNCH(2, 1, 4);
        }
        if (hr == 4) AR_LAUNCH(4, 4, 2);
        if (hr == 2) AR_LAUNCH(4, 2, 4);
        AR_LAUNCH(4, 1, 4);
#undef AR_LAUNCH
    }
    if (act_dtype == GI_DTYPE_F32)
        return launch_generic<float>(q, k_pool, v_pool, block_table, tok_pos, tok_slot, out, n_tokens, n_q, n_kv, d,
                                     page_size, max_pages, n_pool_pages, window, scale, sinks, sink_dtype, d_v, status,
                                     chunk, n_vh, v_row, maps, out_f32, dist_bias, n_dist, means, keep_first, s);
    if (act_dtype == GI_DTYPE_BF16)
        return launch_generic<bf16>(q, k_pool, v_pool, block_table, tok_pos, tok_slot, out, n_tokens, n_q, n_kv, d,
                                    page_size, max_pages, n_pool_pages, window, scale, sinks, sink_dtype, d_v, status,
                                    chunk, n_vh, v_row, maps, out_f32, dist_bias, n_dist, means, keep_first, s);
    GI_REQUIRE(false, "gi_attention_generic: activation dtype %d", act_dtype);
}

// Plain grouped-query attention: keys and values of one shape, one softmax per head, no chunks.
extern "C" int gi_attention_generic(const void* q, const void* k_pool, const void* v_pool, int act_dtype,
                                    const int* block_table, const int* tok_pos, const int* tok_slot,
                                    void* out, int n_tokens, int n_q, int n_kv, int d, int page_size,
                                    int max_pages, int n_pool_pages, int window, float scale, const void* sinks,
                                    int sink_dtype, int d_v, int* status, int single, void* stream) {
    GI_REQUIRE(d_v > 0 && d_v <= d, "gi_attention_generic: %d value columns of rows of %d", d_v, d);
    return gi_attention_masked(q, k_pool, v_pool, act_dtype, block_table, tok_pos, tok_slot, out, n_tokens, n_q, n_kv, d,
                               page_size, max_pages, n_pool_pages, window, scale, sinks, sink_dtype, d_v, status, 0, n_kv, d,
                               1, nullptr, nullptr, 0, nullptr, nullptr, nullptr, 0, 0, 0, 0, 0, single, stream);
}
