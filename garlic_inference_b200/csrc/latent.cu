// Latent attention, the step between the projections and the attention kernel: the new token's latent row
// goes into the paged cache and the queries are put into the form the attention kernel reads.
//
// A token's cache row is [ c (kv_rank) | rotated shared key part (rot_dim) | zeros up to the row's width ],
// c = rmsnorm(first kv_rank columns of the down-projection) * w.  Every head's key is W_uk,h c beside the
// shared rotated part and its value is W_uv,h c, so with q'_h = W_uk,h^T q_h (made by a per-head product
// before this kernel) the score is  q'_h . c + rot(q_rot,h) . rot(k_rot),  attention over the cache rows
// themselves gives sum_j p_j c_j, and W_uv,h is applied to that afterwards: the cache is read once for all
// heads and keys and values are not expanded.  (For long portions of prompts they are, outside this file; the queries are
// then their own unrotated columns beside the rotated part.)
//
// Rotation: pair (2i, 2i+1) of the rotated part (or, in the half layout, pair (i, i + n_rot/2)), i < n_rot / 2,
// turns by the float32 product position * freq[i]; cosine and sine are multiplied by `magnitude`; dimensions from
// n_rot on pass.  The queries may come from a matrix of their own (an up-projection behind a normed latent), and a
// layer that reads another layer's cache rows brings no latent to append (kv_src = null).
// NikolayBlagoev/garlic-inference has one attention (grouped-query, src/models/qwen3/qwen3.cpp:140-179) and
// the rotate-half layout (src/src-cuda/rope.cu:41-79).
#include "common.cuh"
#include <math.h>

// Element j < n_rot of a rotated part `x` after the turn (cs, sn: the pairs' cosines and sines).
template <typename T>
__device__ __forceinline__ float turned(const T* x, int j, int n_rot, int half, const float* cs, const float* sn) {
    if (half) {
        const int h = n_rot >> 1;
        return j < h ? to_f32(x[j]) * cs[j] - to_f32(x[j + h]) * sn[j]
                     : to_f32(x[j]) * cs[j - h] + to_f32(x[j - h]) * sn[j - h];
    }
    const float a = to_f32(x[j & ~1]), b = to_f32(x[j | 1]);
    return (j & 1) ? b * cs[j >> 1] + a * sn[j >> 1] : a * cs[j >> 1] - b * sn[j >> 1];
}

// Queries: row h of a token is [ `lat` columns of q_lat | the rotated part (dr) of q_src | zeros up to q_w ].  q_lat's heads and
// tokens lie lat_hs and lat_ts apart: the dense q' of the absorbed form, or the unrotated columns of q_src themselves.
// A block takes `hpb` heads of a token (one more block per token its cache row), LP_V elements per access when everything
// falls on 16 bytes (the rotated elements a word and its partner word at a time: two-byte loads of both kept the load units
// busy for half of the time).  Measured at 2,048 tokens and 32 heads: rows of 576 92 us element by element with a block, and
// its sines and cosines, per head, 43 us so; rows of 192 21 us.
#define LP_THREADS 128
template <typename T>
__global__ void __launch_bounds__(LP_THREADS)
latent_prepare_kernel(const T* __restrict__ q_src, long long ldq, int q_off,
                      const T* __restrict__ kv_src, long long ld, int c_off, int half,
                      const T* __restrict__ q_lat, long long lat_ts, long long lat_hs, int lat, int q_w, int hpb, int vec,
                      const void* __restrict__ norm_w, int w_dtype,
                      float eps, const float* __restrict__ freq, float magnitude, int n_rot,
                      const int* __restrict__ tok_pos, const int* __restrict__ tok_slot,
                      const int* __restrict__ block_table, T* __restrict__ pool,
                      T* __restrict__ q_out, int H, int d, int dr, int rank, int row_w,
                      int page_size, int max_pages, int n_pool_pages, int append,
                      int* __restrict__ status) {
    gi_pdl_start();
    __shared__ float red[33];
    __shared__ float cs_s[128], sn_s[128];             // cosine and sine of the token's angles, pairs 0 .. n_rot/2 - 1
    const int t = blockIdx.x, part = blockIdx.y;       // part < groups: those heads' query rows; the last one: the cache row
    const int pos = tok_pos[t], slot = tok_slot[t];
    const float p = (float)pos;
    for (int i = threadIdx.x; i < n_rot / 2; i += blockDim.x) {
        float sn, cs;
        sincosf(p * freq[i], &sn, &cs);
        cs_s[i] = cs * magnitude; sn_s[i] = sn * magnitude;
    }
    __syncthreads();

    if (part < (H + hpb - 1) / hpb) {
        constexpr int V = 16 / (int)sizeof(T);
        const int h0 = part * hpb, heads = min(hpb, H - h0), step = vec ? V : 1;
        for (int i = threadIdx.x * step; i < heads * q_w; i += LP_THREADS * step) {
            const int h = h0 + i / q_w, c = i % q_w;
            const T* qr = q_src + (size_t)t * ldq + q_off + (size_t)h * (d + dr) + d;
            const T* ql = q_lat + (size_t)t * lat_ts + (size_t)h * lat_hs;
            T* dst = q_out + ((size_t)t * H + h) * q_w + c;
            if (vec && c < lat) {
                *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<const uint4*>(ql + c);
                continue;
            }
            __align__(16) T v[V];
            if (vec == 2 && c - lat + V <= n_rot) {      // a whole word of rotated elements and the word they turn with
                const int j = c - lat, hh = n_rot >> 1, lower = j < hh;
                const int a0 = half ? (lower ? j : j - hh) : j >> 1;
                __align__(16) T x[V], y[V];
                *reinterpret_cast<uint4*>(x) = *reinterpret_cast<const uint4*>(qr + j);
                if (half) *reinterpret_cast<uint4*>(y) = *reinterpret_cast<const uint4*>(qr + (lower ? j + hh : j - hh));
#pragma unroll
                for (int e = 0; e < V; ++e) {
                    const int a = a0 + (half ? e : e >> 1);
                    const float other = half ? (lower ? -to_f32(y[e]) : to_f32(y[e])) : ((e & 1) ? to_f32(x[e ^ 1]) : -to_f32(x[e ^ 1]));
                    v[e] = from_f32<T>(to_f32(x[e]) * cs_s[a] + other * sn_s[a]);
                }
                *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<const uint4*>(v);
                continue;
            }
#pragma unroll
            for (int e = 0; e < V; ++e) {
                const int j = c + e - lat;
                v[e] = from_f32<T>(0.f);
                if (e < step) {
                    if (j < 0) v[e] = ql[c + e];
                    else if (j < dr) v[e] = from_f32<T>(j < n_rot ? turned(qr, j, n_rot, half, cs_s, sn_s) : to_f32(qr[j]));
                }
            }
            if (vec) *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<const uint4*>(v);
            else *dst = v[0];
        }
        return;
    }
    if (!append || slot < 0 || !kv_src) return;
    const int lp = pos / page_size;
    if (pos < 0 || lp >= max_pages) { if (threadIdx.x == 0) atomicExch(status, 1); return; }
    const int page = block_table[(size_t)slot * max_pages + lp];
    if (page < 0 || page >= n_pool_pages) { if (threadIdx.x == 0) atomicExch(status, 2); return; }
    T* dst = pool + ((size_t)page * page_size + (pos - lp * page_size)) * row_w;

    const T* cr = kv_src + (size_t)t * ld + c_off;
    float ss = 0.f;
#pragma unroll 4
    for (int c = threadIdx.x; c < rank; c += blockDim.x) { const float x = to_f32(cr[c]); ss += x * x; }
    ss = block_sum(ss, red);
    const float inv = 1.f / sqrtf(ss / (float)rank + eps);
#pragma unroll 4
    for (int c = threadIdx.x; c < row_w; c += blockDim.x) {
        float v = 0.f;
        if (c < rank) {
            v = to_f32(cr[c]) * inv * load_w(norm_w, w_dtype, c);
        } else if (c < rank + dr) {
            const int j = c - rank;
            const T* kr = cr + rank;
            v = j < n_rot ? turned(kr, j, n_rot, half, cs_s, sn_s) : to_f32(kr[j]);
        }
        dst[c] = from_f32<T>(v);
    }
}

// q_lat null: the unrotated columns of q_src take its place, rows of d + dr.
extern "C" int gi_latent_prepare(const void* q_src, long long ldq, int q_off, const void* kv_src, long long ld, int c_off,
                                 int half, const void* q_lat,
                                 int act_dtype, const void* norm_w, int w_dtype, float eps, const float* freq,
                                 float magnitude, int n_rot, const int* tok_pos, const int* tok_slot,
                                 const int* block_table, void* pool, void* q_out, int n_tokens, int H, int d, int dr,
                                 int rank, int row_w, int page_size, int max_pages, int n_pool_pages, int append,
                                 int* status, void* stream) {
    GI_REQUIRE(n_tokens >= 0 && H > 0 && d > 0 && dr >= 0 && rank > 0, "gi_latent_prepare: sizes must be positive");
    GI_REQUIRE(row_w >= rank + dr, "gi_latent_prepare: cache rows of %d hold no latent of %d and key part of %d",
               row_w, rank, dr);
    GI_REQUIRE(n_rot % 2 == 0 && n_rot <= dr && n_rot <= 256, "gi_latent_prepare: %d rotated dimensions of %d (at most 256)", n_rot, dr);
    GI_REQUIRE(H < 65535, "gi_latent_prepare: %d heads", H);
    GI_REQUIRE(kv_src || !append, "gi_latent_prepare: nothing to append without a latent of the layer's own");
    GI_REQUIRE(act_dtype == GI_DTYPE_F32 || act_dtype == GI_DTYPE_BF16, "gi_latent_prepare: activation dtype %d", act_dtype);
    if (n_tokens == 0) return 0;
    cudaStream_t s = (cudaStream_t)stream;
    const int item = act_dtype == GI_DTYPE_F32 ? 4 : 2, v = 16 / item;
    const void* src = q_lat ? q_lat : (const unsigned char*)q_src + (size_t)q_off * item;
    const long long lat_ts = q_lat ? (long long)H * rank : ldq, lat_hs = q_lat ? rank : d + dr;
    const int lat = q_lat ? rank : d, q_w = q_lat ? row_w : d + dr;
    // words of 16 bytes: the copied columns (1), and the rotated ones too (2)
    int vec = lat % v == 0 && q_w % v == 0 && lat_ts % v == 0 && lat_hs % v == 0 && (uintptr_t)src % 16 == 0 && (uintptr_t)q_out % 16 == 0;
    if (vec && d % v == 0 && dr % v == 0 && q_off % v == 0 && ldq % v == 0 && (uintptr_t)q_src % 16 == 0 && (!half || n_rot / 2 % v == 0)) vec = 2;
    // prompts: sixteen heads to a block, so that a block moves several KB; few tokens: one, so that every SM gets some
    const int hpb = n_tokens >= 64 ? 16 : 1;
    dim3 grid(n_tokens, (H + hpb - 1) / hpb + 1);
#define LP_LAUNCH(T)                                                                                                            \
    gi_launch(latent_prepare_kernel<T>, grid, dim3(LP_THREADS), 0, s, (const T*)q_src, ldq, q_off, (const T*)kv_src, ld, c_off, half, \
              (const T*)src, lat_ts, lat_hs, lat, q_w, hpb, vec, norm_w, w_dtype, eps, freq, magnitude, n_rot, tok_pos, tok_slot,     \
              block_table, (T*)pool, (T*)q_out, H, d, dr, rank, row_w, page_size, max_pages, n_pool_pages, append, status)
    if (act_dtype == GI_DTYPE_F32) LP_LAUNCH(float);
    else LP_LAUNCH(bf16);
#undef LP_LAUNCH
    return gi_check_launch("gi_latent_prepare");
}

// ------------------------------------------------------------------ both latents of a token whose heads have no rotated part
// The queries' latent, RMS-normed into dense rows, and the keys' and values' latent, RMS-normed into the token's cache
// row (zeros up to the row's width): one launch, blockIdx.y = 0 / 1.  The thread count depends on the wider rank alone
// and sums run in a fixed order, so a row's result does not depend on what else is in the launch.  Four elements per
// access when everything falls on words of four.
template <typename T>
__global__ void latent_norms_kernel(const T* __restrict__ src, long long ld, int q_off, int c_off, const void* __restrict__ q_w,
                                    const void* __restrict__ c_w, int w_dtype, float eps, const int* __restrict__ tok_pos,
                                    const int* __restrict__ tok_slot, const int* __restrict__ block_table, T* __restrict__ pool,
                                    T* __restrict__ q_out, int q_rank, int rank, int row_w, int page_size, int max_pages,
                                    int n_pool_pages, int vec, int* __restrict__ status) {
    gi_pdl_start();
    __shared__ float red[33];
    const int t = blockIdx.x;
    const bool is_q = blockIdx.y == 0;
    const int n = is_q ? q_rank : rank;
    const T* x = src + (size_t)t * ld + (is_q ? q_off : c_off);
    const void* w = is_q ? q_w : c_w;
    T* dst = q_out + (size_t)t * q_rank;
    if (!is_q) {
        const int pos = tok_pos[t], slot = tok_slot[t];
        if (slot < 0) return;
        const int lp = pos >= 0 ? pos / page_size : max_pages;
        if (lp >= max_pages) { if (threadIdx.x == 0) atomicExch(status, 1); return; }
        const int page = block_table[(size_t)slot * max_pages + lp];
        if (page < 0 || page >= n_pool_pages) { if (threadIdx.x == 0) atomicExch(status, 2); return; }
        dst = pool + ((size_t)page * page_size + (pos - lp * page_size)) * row_w;
        for (int c = rank + threadIdx.x; c < row_w; c += blockDim.x) dst[c] = from_f32<T>(0.f);
    }
    float ss = 0.f;
    if (vec) {
        for (int c = threadIdx.x * 4; c < n; c += blockDim.x * 4) {
            const float4 v = load4_act(x + c);
            ss += v.x * v.x; ss += v.y * v.y; ss += v.z * v.z; ss += v.w * v.w;
        }
    } else {
        for (int c = threadIdx.x; c < n; c += blockDim.x) { const float v = to_f32(x[c]); ss += v * v; }
    }
    const float inv = 1.f / sqrtf(block_sum(ss, red) / (float)n + eps);
    if (vec) {
        for (int c = threadIdx.x * 4; c < n; c += blockDim.x * 4) {
            const float4 v = load4_act(x + c), f = load4_w(w, w_dtype, c);
            store4_act(dst + c, make_float4(v.x * inv * f.x, v.y * inv * f.y, v.z * inv * f.z, v.w * inv * f.w));
        }
    } else {
        for (int c = threadIdx.x; c < n; c += blockDim.x) dst[c] = from_f32<T>(to_f32(x[c]) * inv * load_w(w, w_dtype, c));
    }
}

extern "C" int gi_latent_norms(const void* src, long long ld, int q_off, int c_off, int act_dtype, const void* q_w,
                               const void* c_w, int w_dtype, float eps, const int* tok_pos, const int* tok_slot,
                               const int* block_table, void* pool, void* q_out, int n_tokens, int q_rank, int rank, int row_w,
                               int page_size, int max_pages, int n_pool_pages, int* status, void* stream) {
    GI_REQUIRE(n_tokens >= 0 && q_rank > 0 && rank > 0 && row_w >= rank && page_size > 0 && max_pages > 0, "gi_latent_norms: sizes must be positive");
    if (n_tokens == 0) return 0;
    cudaStream_t s = (cudaStream_t)stream;
    const int wide = q_rank > rank ? q_rank : rank, wsz = w_dtype == GI_DTYPE_F32 ? 16 : 8, asz = act_dtype == GI_DTYPE_F32 ? 16 : 8;
    const int threads = wide > 512 ? 256 : (wide > 256 ? 128 : 64);
    const int vec = q_rank % 4 == 0 && rank % 4 == 0 && row_w % 4 == 0 && ld % 4 == 0 && q_off % 4 == 0 && c_off % 4 == 0 &&
                    (uintptr_t)src % asz == 0 && (uintptr_t)pool % asz == 0 && (uintptr_t)q_out % asz == 0 &&
                    (uintptr_t)q_w % wsz == 0 && (uintptr_t)c_w % wsz == 0;
#define LN_LAUNCH(T)                                                                                                    \
    gi_launch(latent_norms_kernel<T>, dim3(n_tokens, 2), dim3(threads), 0, s, (const T*)src, ld, q_off, c_off, q_w, c_w, \
              w_dtype, eps, tok_pos, tok_slot, block_table, (T*)pool, (T*)q_out, q_rank, rank, row_w, page_size, max_pages, \
              n_pool_pages, vec, status)
    if (act_dtype == GI_DTYPE_F32) LN_LAUNCH(float);
    else if (act_dtype == GI_DTYPE_BF16) LN_LAUNCH(bf16);
    else GI_REQUIRE(false, "gi_latent_norms: activation dtype %d", act_dtype);
#undef LN_LAUNCH
    return gi_check_launch("gi_latent_norms");
}

// ------------------------------------------------------------------ attention of single tokens over the latent rows
// Decode steps in bfloat16: one new token per sequence, all heads of a sequence read the same cached rows.  A
// block takes one token, up to 8 * HPW heads and one slice of the keys; it stages 32 rows at a time in shared
// memory, where every head's scores and weighted sums read them (the exact-order kernel fetches them once per
// head).  The slices are of one length over all sequences (ld_slice): a step's sequences are of all lengths, and its longest
// would otherwise keep a few blocks at work when the others have left.  Warp w owns heads w HPW .. w HPW + HPW - 1 of the block's group for all keys of the slice, so the
// running maximum and sum stay inside the warp; lane j scores key j of the 32, then the lanes turn to pairs of
// value columns.  Scores, softmax and sums are float32.  The slices' (max, sum, weighted rows) go to `part`
// [blocks, heads, 2 + rank] and latent_decode_combine_kernel merges them with the sink.
#define LD_WARPS 8
#define LD_KEYS 32

// chunks of 32 keys that token t sees, 0 for a row that is none (a recorded step's padding)
__device__ __forceinline__ int ld_chunks(int t, const int* __restrict__ tok_pos, const int* __restrict__ tok_slot, int page_size,
                                         int max_pages, int window, bool& bad) {
    const int slot = tok_slot[t], pos = tok_pos[t];
    if (slot < 0 || pos < 0 || pos / page_size >= max_pages) {
        bad = bad || slot >= 0;
        return 0;
    }
    return pos / LD_KEYS - (window > 0 ? max(0, pos - window + 1) : 0) / LD_KEYS + 1;
}

// Which token's slice, of how many, block b of `n_blocks` takes (n_blocks >= n_tokens).  Up to LD_SLICED tokens: every token's chunks are cut into the
// fewest slices of at most `per` chunks, `per` the least (from `least` on) with which all tokens' slices are no more than the blocks.  Beyond, where
// every one of so many blocks would search for longer than that evens out: as many slices of each, n_blocks / n_tokens.  t = -1: none.  From
// positions and slots alone, before the kernel ahead has finished: a thread looks a token up, warp 0 searches with them in registers.
// Measured in a recorded step, 32 heads over rows of 576, us with the tokens looked up in every pass of the search and no limit / so: 1 sequence
// of 20 tokens 15.5 / 13.9, 64 of 200 to 4,000 112 / 109, 128 of 100 41.6 / 36.9, 256 of 100 93 / 50, 1,000 of 50 to 600 833 / 294; a slice or
// more of its own length for every sequence 20.5, 186, 39.7, 56, 343.
#define LD_SLICED (LD_WARPS * 32)
struct LdSlice { int t, split, n_splits; };
struct LdFind { LdSlice mine; int chunks[LD_SLICED]; };
__host__ __device__ __forceinline__ int2* ld_table(float* part, size_t floats) { return reinterpret_cast<int2*>(part + (floats + 1) / 2 * 2); }
// ceil(a / b) for many a: by a multiplication where that is exact (a + b below 2^16, two million positions)
struct LdCeil {
    int b;
    unsigned scale;
    __device__ __forceinline__ LdCeil(int b_, int most) : b(b_), scale(most + b_ < 65536 ? 0xffffffffu / b_ + 1 : 0u) {}
    __device__ __forceinline__ int operator()(int a) const {
        return b == 1 ? a : scale ? (int)__umulhi(a + b - 1, scale) : (int)(((long long)a + b - 1) / b);
    }
};
// first[i], count[i]: first block and slices of token 32 i + lane, for the table
__device__ __forceinline__ void ld_find_slice(int b, int n_blocks, int n_tokens, int least, LdFind* find, int (&first)[LD_SLICED / 32],
                                              int (&count)[LD_SLICED / 32]) {
    const int lane = threadIdx.x;
    int total = 0, live = 0, most = 0;
#pragma unroll
    for (int i = 0; i < LD_SLICED / 32; ++i) {
        if (i * 32 >= n_tokens) break;
        count[i] = i * 32 + lane < n_tokens ? find->chunks[i * 32 + lane] : 0;
        total += count[i];
        live += count[i] > 0;
        most = max(most, count[i]);
    }
    total = __reduce_add_sync(0xffffffffu, total);
    live = __reduce_add_sync(0xffffffffu, live);
    most = __reduce_max_sync(0xffffffffu, most);
    int per = max(least, (total + n_blocks - 1) / n_blocks);
    int enough = min(max(1, most), max(per, n_blocks > live ? (total + n_blocks - live - 1) / (n_blocks - live) : most));
    per = min(per, enough);
    while (per < enough) {
        const LdCeil slices((per + enough) / 2, most);
        int n = 0;
#pragma unroll
        for (int i = 0; i < LD_SLICED / 32; ++i) {
            if (i * 32 >= n_tokens) break;
            n += slices(count[i]);
        }
        if (__reduce_add_sync(0xffffffffu, n) <= n_blocks) enough = slices.b;
        else per = slices.b + 1;
    }
    if (lane == 0) find->mine.t = -1;
    __syncwarp();
    const LdCeil slices(per, most);
    int base = 0;
#pragma unroll
    for (int i = 0; i < LD_SLICED / 32; ++i) {
        if (i * 32 >= n_tokens) break;
        count[i] = slices(count[i]);
        int end = count[i];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int x = __shfl_up_sync(0xffffffffu, end, o);
            if (lane >= o) end += x;
        }
        first[i] = base + end - count[i];
        if (b >= first[i] && b < first[i] + count[i]) find->mine = {i * 32 + lane, b - first[i], count[i]};
        base += __shfl_sync(0xffffffffu, end, 31);
    }
}

// By a whole block; waits for the kernel ahead, and writes {first block, slices} of every token to the table.
__device__ __forceinline__ LdSlice ld_slice(int n_blocks, int n_tokens, int least, const int* __restrict__ tok_pos, const int* __restrict__ tok_slot,
                                            int page_size, int max_pages, int window, int2* table, int* status, LdFind* find) {
    gi_pdl_launch_dependents();
    const int b = blockIdx.x, tid = threadIdx.x;
    bool bad = false;                            // a row beyond its page table
    if (n_tokens > LD_SLICED) {
        const int each = n_blocks / n_tokens, t = b / each;
        const int chunks = t < n_tokens ? ld_chunks(t, tok_pos, tok_slot, page_size, max_pages, window, bad) : 0;
        const LdSlice s = {b % each < chunks ? t : -1, b % each, min(each, chunks)};
        gi_pdl_wait();
        if (t < n_tokens && s.split == 0 && blockIdx.y == 0 && tid == 0) {
            table[t] = make_int2(b, s.n_splits);
            if (bad) atomicExch(status, 4);
        }
        return s;
    }
    if (tid < n_tokens) find->chunks[tid] = ld_chunks(tid, tok_pos, tok_slot, page_size, max_pages, window, bad);
    __syncthreads();
    int first[LD_SLICED / 32], count[LD_SLICED / 32];
    if (tid < 32) ld_find_slice(b, n_blocks, n_tokens, least, find, first, count);
    gi_pdl_wait();
    if (b == 0 && blockIdx.y == 0) {
        if (tid < 32) {
#pragma unroll
            for (int i = 0; i < LD_SLICED / 32; ++i)
                if (i * 32 + tid < n_tokens) table[i * 32 + tid] = make_int2(first[i], count[i]);
        }
        if (bad) atomicExch(status, 4);
    }
    __syncthreads();
    return find->mine;
}

// A block's slice: t, slot, pos, its chunks c0 .. c1 - 1, first seen key lo, its results at `my`.
#define LD_FIND_SLICE                                                                                                            \
    __shared__ LdFind ld_mine;                                                                                                   \
    const LdSlice ld_s = ld_slice(n_blocks, n_tokens, least, tok_pos, tok_slot, page_size, max_pages, window,                    \
                                  ld_table(part, (size_t)n_blocks * H * stride), status, &ld_mine);                             \
    if (ld_s.t < 0) return;                                                                                                      \
    const int t = ld_s.t, slot = tok_slot[t], pos = tok_pos[t], lo = window > 0 ? max(0, pos - window + 1) : 0;                  \
    const int ld_n = pos / LD_KEYS - lo / LD_KEYS + 1;                                                                           \
    const int c0 = lo / LD_KEYS + (int)((long long)ld_n * ld_s.split / ld_s.n_splits);                                           \
    const int c1 = lo / LD_KEYS + (int)((long long)ld_n * (ld_s.split + 1) / ld_s.n_splits);                                     \
    float* my = part + (size_t)blockIdx.x * H * stride;

// What a chunk's exponents are taken from: the maximum, which is minus infinity while all scores are (every chunk holds a seen key, but its
// score may be beyond the finite): their weights are zero then.
__device__ __forceinline__ float ld_from(float maximum) { return maximum == -INFINITY ? 0.f : maximum; }

__device__ __forceinline__ float2 bf2_to_f2(uint32_t w) {
    return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w));
}

template <int HPW, int DPL2>
__global__ void __launch_bounds__(LD_WARPS * 32)
latent_decode_kernel(const bf16* __restrict__ q, const bf16* __restrict__ pool, const int* __restrict__ block_table,
                     const int* __restrict__ tok_pos, const int* __restrict__ tok_slot, float* __restrict__ part,
                     int H, int dk, int rank, int page_size, int max_pages, int n_pool_pages, int n_blocks, int n_tokens, int least,
                     float scale, int* __restrict__ status, int window) {
    extern __shared__ __align__(16) unsigned char ld_smem[];
    constexpr int HG = HPW * LD_WARPS;
    float* q_s = reinterpret_cast<float*>(ld_smem);                  // HG rows of dk
    uint32_t* k_s = reinterpret_cast<uint32_t*>(q_s + HG * dk);      // 32 rows of kw words (kw odd: no bank conflicts)
    const int kw = dk / 2 + 1;
    const size_t stride = (size_t)rank + 2;
    LD_FIND_SLICE
    const int h0 = blockIdx.y * HG;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

        for (int i = threadIdx.x; i < HG * dk; i += blockDim.x) {
            const int hh = i / dk, c = i - hh * dk;
            q_s[i] = h0 + hh < H ? to_f32(q[((size_t)t * H + h0 + hh) * dk + c]) * scale : 0.f;
        }
    float m[HPW], l[HPW], p[HPW], acc[HPW][2 * DPL2];
#pragma unroll
    for (int hh = 0; hh < HPW; ++hh) {
        m[hh] = -INFINITY; l[hh] = 0.f;
#pragma unroll
        for (int r = 0; r < 2 * DPL2; ++r) acc[hh][r] = 0.f;
    }
    const int* bt = block_table + (size_t)slot * max_pages;
    const int vec_per_row = dk / 8;
    for (int c = c0; c < c1; ++c) {
        __syncthreads();
        for (int idx = threadIdx.x; idx < LD_KEYS * vec_per_row; idx += blockDim.x) {
            const int j = idx / vec_per_row, v = idx - j * vec_per_row;
            const int key = c * LD_KEYS + j;
            uint4 val = make_uint4(0u, 0u, 0u, 0u);
            if (key >= lo && key <= pos) {
                const int page = bt[key / page_size];
                if (page < 0 || page >= n_pool_pages) atomicExch(status, 5);
                else val = *reinterpret_cast<const uint4*>(pool + ((size_t)page * page_size + key % page_size) * dk + v * 8);
            }
            uint32_t* dst = k_s + j * kw + v * 4;
            dst[0] = val.x; dst[1] = val.y; dst[2] = val.z; dst[3] = val.w;
        }
        __syncthreads();
        const bool valid = c * LD_KEYS + lane >= lo && c * LD_KEYS + lane <= pos;
        float s[HPW];
#pragma unroll
        for (int hh = 0; hh < HPW; ++hh) s[hh] = 0.f;
        const uint32_t* kr = k_s + lane * kw;
        const float* qw = q_s + (size_t)warp * HPW * dk;
        for (int i2 = 0; i2 < dk / 2; ++i2) {
            const float2 kf = bf2_to_f2(kr[i2]);
#pragma unroll
            for (int hh = 0; hh < HPW; ++hh) {
                const float2 qf = *reinterpret_cast<const float2*>(qw + hh * dk + 2 * i2);
                s[hh] = fmaf(kf.x, qf.x, s[hh]);
                s[hh] = fmaf(kf.y, qf.y, s[hh]);
            }
        }
#pragma unroll
        for (int hh = 0; hh < HPW; ++hh) {
            const float sv = valid ? s[hh] : -INFINITY;
            const float m_new = fmaxf(m[hh], warp_max(sv)), from = ld_from(m_new);
            const float corr = expf(m[hh] - from);
            p[hh] = valid ? expf(sv - from) : 0.f;
            l[hh] = l[hh] * corr + warp_sum(p[hh]);
            m[hh] = m_new;
#pragma unroll
            for (int r = 0; r < 2 * DPL2; ++r) acc[hh][r] *= corr;
        }
        for (int j = 0; j < LD_KEYS; ++j) {
            float pj[HPW];
#pragma unroll
            for (int hh = 0; hh < HPW; ++hh) pj[hh] = __shfl_sync(0xffffffffu, p[hh], j);
#pragma unroll
            for (int r = 0; r < DPL2; ++r) {
                const int col2 = lane + 32 * r;
                if (2 * col2 < rank) {
                    const float2 vf = bf2_to_f2(k_s[j * kw + col2]);
#pragma unroll
                    for (int hh = 0; hh < HPW; ++hh) {
                        acc[hh][2 * r] = fmaf(pj[hh], vf.x, acc[hh][2 * r]);
                        acc[hh][2 * r + 1] = fmaf(pj[hh], vf.y, acc[hh][2 * r + 1]);
                    }
                }
            }
        }
    }
#pragma unroll
    for (int hh = 0; hh < HPW; ++hh) {
        const int h = h0 + warp * HPW + hh;
        if (h >= H) continue;
        float* o = my + (size_t)h * stride;
        if (lane == 0) { o[0] = m[hh]; o[1] = l[hh]; }
#pragma unroll
        for (int r = 0; r < DPL2; ++r) {
            const int col = 2 * (lane + 32 * r);
            if (col < rank) o[2 + col] = acc[hh][2 * r];
            if (col + 1 < rank) o[2 + col + 1] = acc[hh][2 * r + 1];
        }
    }
}

// The same block on tensor cores (mma.sync m16n8k16, bfloat16 operands, float32 accumulation).  A block takes
// 32 heads: the scores of a chunk, 32 heads x 32 keys, are 2 x 4 tiles, one per warp, summed over the row's
// width in steps of 16; they go through shared memory as float32 to the softmax (warp w owns heads 4w .. 4w+3,
// as above: maximum, sum and weights float32); the weights, rounded to bfloat16 as the second product's
// operand, times the staged rows' first `rank` columns are 2 x ceil(rank / 8) tiles, NTW column tiles per
// warp, with the rows read as the product's second operand by ldmatrix.trans.  Shared-memory rows are padded
// to 4 words past a multiple of 32 so that the fragments' loads meet no bank twice.
__device__ __forceinline__ void mma_bf16_16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// Two blocks fit an SM: one's copies and barriers run under the other's products, so a block stages one chunk at a time.  A
// chunk costs its block a serial chain (copy, scores, softmax, weighted rows); the scores' steps therefore go in two
// sums of half the width each, their fragments four steps ahead.  Measured with 20 sequences of 200 to 4,000 tokens, 32 heads,
// rows of 576 (a recorded step has 32 rows), in 8 slices: 112 us before both and before the look-ups were a warp's, 93 us so;
// 64 sequences of 2,048 in 4 slices 214 -> 115 us.
template <int NTW>
__global__ void __launch_bounds__(LD_WARPS * 32, 2)
latent_decode_mma_kernel(const bf16* __restrict__ q, const bf16* __restrict__ pool, const int* __restrict__ block_table,
                         const int* __restrict__ tok_pos, const int* __restrict__ tok_slot, float* __restrict__ part,
                         int H, int dk, int rank, int row_words, int page_size, int max_pages, int n_pool_pages,
                         int n_blocks, int n_tokens, int least, float scale, int* __restrict__ status, int window) {
    extern __shared__ __align__(16) unsigned char ld_smem[];
    constexpr int HG = 32, PW = 20;                                  // heads per block; words per row of weights
    const int kw = row_words;                                        // words per staged row, kw % 32 == 4
    uint32_t* q_b = reinterpret_cast<uint32_t*>(ld_smem);            // HG rows of kw words (bfloat16 pairs)
    uint32_t* k_s = q_b + HG * kw;                                   // 32 rows of kw words
    float* s_s = reinterpret_cast<float*>(k_s + LD_KEYS * kw);       // HG x 33 scores
    uint32_t* p_s = reinterpret_cast<uint32_t*>(s_s + HG * 33);      // HG rows of PW words: the weights
    float* corr_s = reinterpret_cast<float*>(p_s + HG * PW);         // HG
    const size_t stride = (size_t)rank + 2;
    LD_FIND_SLICE
    const int h0 = blockIdx.y * HG;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, tq = lane & 3;                          // the fragments' row group and column pair
    const int vec_per_row = dk / 8, words = dk / 2;

    for (int idx = threadIdx.x; idx < HG * (kw / 4); idx += blockDim.x) {
        const int hh = idx / (kw / 4), v = idx - hh * (kw / 4);
        uint4 val = make_uint4(0u, 0u, 0u, 0u);
        if (h0 + hh < H && v < vec_per_row)
            val = *reinterpret_cast<const uint4*>(q + ((size_t)t * H + h0 + hh) * dk + v * 8);
        *reinterpret_cast<uint4*>(q_b + hh * kw + v * 4) = val;
    }
    float m[4], l[4];
#pragma unroll
    for (int hh = 0; hh < 4; ++hh) { m[hh] = -INFINITY; l[hh] = 0.f; }
    float acc[2][NTW][4];
#pragma unroll
    for (int mt = 0; mt < 2; ++mt)
#pragma unroll
        for (int j = 0; j < NTW; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[mt][j][e] = 0.f;
    const int* bt = block_table + (size_t)slot * max_pages;
    const int k_steps = (words + 7) / 8;                              // steps of 16 values; the rows' padding is zero
    const int mt_s = warp & 1, nt_s = warp >> 1;                      // this warp's tile of the scores
    const int n_tiles = (rank + 7) / 8;
    const uint32_t k_s_addr = (uint32_t)__cvta_generic_to_shared(k_s);
    // Asynchronous 16-byte copies of a chunk's rows, four rows to a warp; keys out of sight, unmapped pages and
    // the rows' padding are filled with zeros (a copy of 0 source bytes).  Lane r < 4 looks up where the warp's row r of the
    // next chunk lies while this one is walked.  (A division for each copy's row, column and page took most of a chunk's time.)
    auto where = [&](int c) -> long long {                            // first element of this lane's row, or -1: zeros
        const int key = c * LD_KEYS + warp * 4 + lane;
        if (lane >= 4 || c >= c1 || key < lo || key > pos) return -1;
        const int lp = key / page_size, page = bt[lp];
        if (page < 0 || page >= n_pool_pages) { atomicExch(status, 5); return -1; }
        return ((long long)page * page_size + (key - lp * page_size)) * dk;
    };
    long long next = where(c0);
    auto stage = [&](int c) {
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const long long at = __shfl_sync(0xffffffffu, next, r);
            const uint32_t dst = k_s_addr + (warp * 4 + r) * kw * 4;
            for (int v = lane; v < kw / 4; v += 32) {
                const int bytes = at >= 0 && v < vec_per_row ? 16 : 0;
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" :: "r"(dst + v * 16), "l"(pool + (bytes ? at + v * 8 : 0)), "r"(bytes) : "memory");
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        next = where(c + 1);
    };

    for (int c = c0; c < c1; ++c) {
        __syncthreads();                                              // the last chunk's rows and weights are done with
        stage(c);
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        // scores: tile (mt_s, nt_s) = heads 16 mt_s .. +15 x keys 8 nt_s .. +7
        {
            float sc[4] = {0.f, 0.f, 0.f, 0.f}, sd[4] = {0.f, 0.f, 0.f, 0.f};
            const uint32_t* qa = q_b + (16 * mt_s + g) * kw + tq;
            const uint32_t* kb = k_s + (8 * nt_s + g) * kw + tq;
            int ks = 0;
            for (; ks + 4 <= k_steps; ks += 4) {
                uint32_t a[4][4], b[4][2];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const int at = 8 * (ks + u);
                    a[u][0] = qa[at]; a[u][1] = qa[8 * kw + at]; a[u][2] = qa[at + 4]; a[u][3] = qa[8 * kw + at + 4];
                    b[u][0] = kb[at]; b[u][1] = kb[at + 4];
                }
                mma_bf16_16816(sc, a[0], b[0][0], b[0][1]);
                mma_bf16_16816(sd, a[1], b[1][0], b[1][1]);
                mma_bf16_16816(sc, a[2], b[2][0], b[2][1]);
                mma_bf16_16816(sd, a[3], b[3][0], b[3][1]);
            }
            for (; ks < k_steps; ++ks) {
                const uint32_t a[4] = {qa[8 * ks], qa[8 * kw + 8 * ks], qa[8 * ks + 4], qa[8 * kw + 8 * ks + 4]};
                mma_bf16_16816(sc, a, kb[8 * ks], kb[8 * ks + 4]);
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) sc[e] += sd[e];
            float* srow = s_s + (16 * mt_s + g) * 33 + 8 * nt_s + 2 * tq;
            srow[0] = sc[0] * scale; srow[1] = sc[1] * scale;
            srow[8 * 33] = sc[2] * scale; srow[8 * 33 + 1] = sc[3] * scale;
        }
        __syncthreads();
        // softmax of the chunk: warp w owns heads 4 w .. 4 w + 3, lane j is key j
        {
            const bool valid = c * LD_KEYS + lane >= lo && c * LD_KEYS + lane <= pos;
#pragma unroll
            for (int hh = 0; hh < 4; ++hh) {
                const int h = 4 * warp + hh;
                const float sv = valid ? s_s[h * 33 + lane] : -INFINITY;
                const float m_new = fmaxf(m[hh], warp_max(sv)), from = ld_from(m_new);
                const float corr = expf(m[hh] - from);
                const bf16 pr = __float2bfloat16_rn(valid ? expf(sv - from) : 0.f);
                l[hh] = l[hh] * corr + warp_sum(__bfloat162float(pr));
                m[hh] = m_new;
                reinterpret_cast<bf16*>(p_s + h * PW)[lane] = pr;
                if (lane == 0) corr_s[h] = corr;
            }
        }
        __syncthreads();
        // weighted rows: this warp's NTW column tiles for both halves of the heads
#pragma unroll
        for (int mt = 0; mt < 2; ++mt) {
            const float ca = corr_s[16 * mt + g], cb = corr_s[16 * mt + g + 8];
#pragma unroll
            for (int j = 0; j < NTW; ++j) { acc[mt][j][0] *= ca; acc[mt][j][1] *= ca; acc[mt][j][2] *= cb; acc[mt][j][3] *= cb; }
        }
#pragma unroll
        for (int ks = 0; ks < 2; ++ks) {
            uint32_t a[2][4];
#pragma unroll
            for (int mt = 0; mt < 2; ++mt) {
                const uint32_t* pa = p_s + (16 * mt + g) * PW + 8 * ks + tq;
                a[mt][0] = pa[0]; a[mt][1] = pa[8 * PW]; a[mt][2] = pa[4]; a[mt][3] = pa[8 * PW + 4];
            }
#pragma unroll
            for (int j = 0; j < NTW; ++j) {
                const int nt = warp * NTW + j;
                if (nt >= n_tiles) continue;                          // uniform over the warp
                uint32_t b0, b1;
                const uint32_t addr = k_s_addr + ((16 * ks + (lane & 15)) * kw + 4 * nt) * 4;
                asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];" : "=r"(b0), "=r"(b1) : "r"(addr));
                mma_bf16_16816(acc[0][j], a[0], b0, b1);
                mma_bf16_16816(acc[1][j], a[1], b0, b1);
            }
        }
    }
    // this slice's (max, sum) of the heads this warp owned in the softmax, and its columns of every head
#pragma unroll
    for (int hh = 0; hh < 4; ++hh) {
        const int h = h0 + 4 * warp + hh;
        if (h < H && lane == 0) { my[(size_t)h * stride] = m[hh]; my[(size_t)h * stride + 1] = l[hh]; }
    }
#pragma unroll
    for (int mt = 0; mt < 2; ++mt)
#pragma unroll
        for (int j = 0; j < NTW; ++j) {
            const int col = 8 * (warp * NTW + j) + 2 * tq;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int h = h0 + 16 * mt + g + (e >> 1) * 8, cc = col + (e & 1);
                if (h < H && cc < rank) my[(size_t)h * stride + 2 + cc] = acc[mt][j][e];
            }
        }
}

// The same for rows of up to 64 KQ values, a block to an SM.  The scores of a chunk are shared out by values: a warp has a quarter of a
// row's, both halves of the heads and one of the keys, so that the queries stay in registers and a staged row is read twice instead of
// four times; the quarters meet in the softmax.  Copies are two chunks ahead.
// Bound by the chain of a chunk (copy, scores, softmax, weighted rows) and its three barriers: the tensor pipe is busy for 15 % of the time, the
// issue slots for 27 %.
// Measured, 32 heads over rows of 576 (the merge included), us with a slice of its own length for every sequence and the kernel above /
// with slices of one length / so: 20 sequences of 200 to 4,000 tokens 79 / 54 / 41, 1 of 2,048 37 / 35 / 25, 8 of 2,048 39 / 37 / 27, 32 of
// 2,048 74 / 66 / 53, 64 of 200 to 4,000 156 / 121 / 112.
#define LW_STAGES 3
#define LW_PER_SM(KQ) ((KQ) == 3 ? 2 : 1)        // blocks to an SM
#define LW_SLD 40            // floats of a row of scores: 8 banks from head to head
template <int KQ, int NTW>
__global__ void __launch_bounds__(LD_WARPS * 32, LW_PER_SM(KQ))
latent_decode_quarters_kernel(const bf16* __restrict__ q, const bf16* __restrict__ pool, const int* __restrict__ block_table,
                              const int* __restrict__ tok_pos, const int* __restrict__ tok_slot, float* __restrict__ part,
                              int H, int dk, int rank, int row_words, int page_size, int max_pages, int n_pool_pages,
                              int n_blocks, int n_tokens, int least, float scale, int* __restrict__ status, int window) {
    extern __shared__ __align__(16) unsigned char ld_smem[];
    constexpr int HG = 32, PW = 20;                                  // heads per block; words per row of weights
    const int kw = row_words;                                        // words per staged row, kw % 32 == 4
    uint32_t* k_s = reinterpret_cast<uint32_t*>(ld_smem);            // [stage][32 rows of kw words]
    float* s_s = reinterpret_cast<float*>(k_s + LW_STAGES * LD_KEYS * kw);       // [quarter][HG][LW_SLD]
    uint32_t* p_s = reinterpret_cast<uint32_t*>(s_s + 4 * HG * LW_SLD);          // HG rows of PW words: the weights
    float* corr_s = reinterpret_cast<float*>(p_s + HG * PW);         // HG
    const size_t stride = (size_t)rank + 2;
    LD_FIND_SLICE
    const int h0 = blockIdx.y * HG;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, tq = lane & 3;                          // the fragments' row group and column pair
    const int* bt = block_table + (size_t)slot * max_pages;
    const int vec_per_row = dk / 8, k_steps = (dk + 15) / 16, per_quarter = (k_steps + 3) / 4;
    const int quarter = warp & 3, keys = warp >> 2;                  // this warp's share of the scores: values, half of the keys
    const int n_tiles = (rank + 7) / 8;
    const uint32_t k_s_addr = (uint32_t)__cvta_generic_to_shared(k_s);
    // Asynchronous 16-byte copies of a chunk's rows, four rows to a warp; keys out of sight, unmapped pages and the rows' padding are
    // filled with zeros.  Lane r < 4 looks up where the warp's row r of the chunk after this one lies.
    auto where = [&](int c) -> long long {                            // first element of this lane's row, or -1: zeros
        const int key = c * LD_KEYS + warp * 4 + lane;
        if (lane >= 4 || c >= c1 || key < lo || key > pos) return -1;
        const int lp = key / page_size, page = bt[lp];
        if (page < 0 || page >= n_pool_pages) { atomicExch(status, 5); return -1; }
        return ((long long)page * page_size + (key - lp * page_size)) * dk;
    };
    long long next = where(c0);
    auto stage = [&](int c) {
        if (c < c1) {
            const uint32_t to = k_s_addr + (uint32_t)((c - c0) % LW_STAGES * LD_KEYS + warp * 4) * kw * 4;
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const long long at = __shfl_sync(0xffffffffu, next, r);
                for (int v = lane; v < kw / 4; v += 32) {
                    const int bytes = at >= 0 && v < vec_per_row ? 16 : 0;
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" :: "r"(to + r * kw * 4 + v * 16), "l"(pool + (bytes ? at + v * 8 : 0)), "r"(bytes) : "memory");
                }
            }
            next = where(c + 1);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");          // an empty group at the end: the count stays uniform
    };
    for (int c = c0; c < c0 + LW_STAGES - 1; ++c) stage(c);
    // the queries' fragments of this warp's values, both halves of the heads
    uint32_t qa[KQ][2][4];
#pragma unroll
    for (int i = 0; i < KQ; ++i)
#pragma unroll
        for (int mt = 0; mt < 2; ++mt)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int h = h0 + 16 * mt + g + (e & 1) * 8, d = (quarter * per_quarter + i) * 16 + 2 * tq + (e >> 1) * 8;
                qa[i][mt][e] = i < per_quarter && h < H && d < dk ? *reinterpret_cast<const uint32_t*>(q + ((size_t)t * H + h) * dk + d) : 0u;
            }
    float m[4], l[4];
#pragma unroll
    for (int hh = 0; hh < 4; ++hh) { m[hh] = -INFINITY; l[hh] = 0.f; }
    float acc[2][NTW][4];
#pragma unroll
    for (int mt = 0; mt < 2; ++mt)
#pragma unroll
        for (int j = 0; j < NTW; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[mt][j][e] = 0.f;

    for (int c = c0; c < c1; ++c) {
        asm volatile("cp.async.wait_group %0;" ::"n"(LW_STAGES - 2) : "memory");
        __syncthreads();                                              // this chunk is there, the one before it is done with
        stage(c + LW_STAGES - 1);
        const uint32_t rows = k_s_addr + (uint32_t)((c - c0) % LW_STAGES * LD_KEYS) * kw * 4;
        {
            float sc[2][2][4] = {};                                   // [half of the heads][8 keys]
            // lanes 0..7, 8..15: 8 keys' first and second 16 bytes of a step of 16 values; 16..31: of the next 8 keys
            const uint32_t from = rows + ((keys * 16 + (lane >> 4) * 8 + (lane & 7)) * kw + (quarter * per_quarter) * 8 + (lane >> 3 & 1) * 4) * 4;
#pragma unroll
            for (int i = 0; i < KQ; ++i) {
                if (i >= per_quarter || quarter * per_quarter + i >= k_steps) break;      // uniform over the warp
                uint32_t b[4];
                asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                             : "=r"(b[0]), "=r"(b[1]), "=r"(b[2]), "=r"(b[3]) : "r"(from + i * 32));
#pragma unroll
                for (int mt = 0; mt < 2; ++mt) {
                    mma_bf16_16816(sc[mt][0], qa[i][mt], b[0], b[1]);
                    mma_bf16_16816(sc[mt][1], qa[i][mt], b[2], b[3]);
                }
            }
#pragma unroll
            for (int mt = 0; mt < 2; ++mt)
#pragma unroll
                for (int nt = 0; nt < 2; ++nt) {
                    float* to = s_s + (quarter * HG + 16 * mt + g) * LW_SLD + keys * 16 + nt * 8 + 2 * tq;
                    *reinterpret_cast<float2*>(to) = make_float2(sc[mt][nt][0], sc[mt][nt][1]);
                    *reinterpret_cast<float2*>(to + 8 * LW_SLD) = make_float2(sc[mt][nt][2], sc[mt][nt][3]);
                }
        }
        __syncthreads();
        // softmax of the chunk: warp w owns heads 4 w .. 4 w + 3, lane j is key j
        {
            const bool valid = c * LD_KEYS + lane >= lo && c * LD_KEYS + lane <= pos;
            float sv[4], mx[4], pr[4];
#pragma unroll
            for (int hh = 0; hh < 4; ++hh) {
                const float* x = s_s + (4 * warp + hh) * LW_SLD + lane;
                const float sum = ((x[0] + x[HG * LW_SLD]) + x[2 * HG * LW_SLD]) + x[3 * HG * LW_SLD];
                sv[hh] = valid ? sum * scale : -INFINITY;
                mx[hh] = sv[hh];
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                for (int hh = 0; hh < 4; ++hh) mx[hh] = fmaxf(mx[hh], __shfl_xor_sync(0xffffffffu, mx[hh], o));
#pragma unroll
            for (int hh = 0; hh < 4; ++hh) {
                const float m_new = fmaxf(m[hh], mx[hh]), from = ld_from(m_new);
                const float corr = expf(m[hh] - from);
                const bf16 w = __float2bfloat16_rn(valid ? expf(sv[hh] - from) : 0.f);
                pr[hh] = __bfloat162float(w);
                l[hh] *= corr;
                m[hh] = m_new;
                reinterpret_cast<bf16*>(p_s + (4 * warp + hh) * PW)[lane] = w;
                if (lane == 0) corr_s[4 * warp + hh] = corr;
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                for (int hh = 0; hh < 4; ++hh) pr[hh] += __shfl_xor_sync(0xffffffffu, pr[hh], o);
#pragma unroll
            for (int hh = 0; hh < 4; ++hh) l[hh] += pr[hh];
        }
        __syncthreads();
        // weighted rows: this warp's NTW column tiles for both halves of the heads
#pragma unroll
        for (int mt = 0; mt < 2; ++mt) {
            const float ca = corr_s[16 * mt + g], cb = corr_s[16 * mt + g + 8];
#pragma unroll
            for (int j = 0; j < NTW; ++j) { acc[mt][j][0] *= ca; acc[mt][j][1] *= ca; acc[mt][j][2] *= cb; acc[mt][j][3] *= cb; }
        }
#pragma unroll
        for (int ks = 0; ks < 2; ++ks) {
            uint32_t a[2][4];
#pragma unroll
            for (int mt = 0; mt < 2; ++mt) {
                const uint32_t* pa = p_s + (16 * mt + g) * PW + 8 * ks + tq;
                a[mt][0] = pa[0]; a[mt][1] = pa[8 * PW]; a[mt][2] = pa[4]; a[mt][3] = pa[8 * PW + 4];
            }
#pragma unroll
            for (int j = 0; j < NTW; j += 2) {
                const int nt = warp * NTW + j;
                if (nt >= n_tiles) continue;                          // uniform over the warp
                // (the second tile's columns lie inside the staged row where it is one of the rank's; else its sums are not stored)
                const uint32_t addr = rows + ((16 * ks + (lane & 15)) * kw + 4 * min(nt + (lane >> 4), n_tiles - 1)) * 4;
                uint32_t b[4];
                asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                             : "=r"(b[0]), "=r"(b[1]), "=r"(b[2]), "=r"(b[3]) : "r"(addr));
                mma_bf16_16816(acc[0][j], a[0], b[0], b[1]);
                mma_bf16_16816(acc[1][j], a[1], b[0], b[1]);
                if (NTW > 1) {
                    mma_bf16_16816(acc[0][(j + 1) % NTW], a[0], b[2], b[3]);
                    mma_bf16_16816(acc[1][(j + 1) % NTW], a[1], b[2], b[3]);
                }
            }
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    // this slice's (max, sum) of the heads this warp owned in the softmax, and its columns of every head
#pragma unroll
    for (int hh = 0; hh < 4; ++hh) {
        const int h = h0 + 4 * warp + hh;
        if (h < H && lane == 0) { my[(size_t)h * stride] = m[hh]; my[(size_t)h * stride + 1] = l[hh]; }
    }
#pragma unroll
    for (int mt = 0; mt < 2; ++mt)
#pragma unroll
        for (int j = 0; j < NTW; ++j) {
            const int col = 8 * (warp * NTW + j) + 2 * tq;
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const int h = h0 + 16 * mt + g + half * 8;
                if (h >= H) continue;
                float* to = my + (size_t)h * stride + 2 + col;
                if (col + 1 < rank && rank % 2 == 0) *reinterpret_cast<float2*>(to) = make_float2(acc[mt][j][2 * half], acc[mt][j][2 * half + 1]);
                else {
                    if (col < rank) to[0] = acc[mt][j][2 * half];
                    if (col + 1 < rank) to[1] = acc[mt][j][2 * half + 1];
                }
            }
        }
}

// Merges a token's slices: a block takes a head's columns, 2 NP to a thread.  table: {first block, slices} of each token.
#define LC_THREADS 128
template <int NP>
__global__ void __launch_bounds__(LC_THREADS)
latent_decode_combine_kernel(const float* __restrict__ part, const int2* __restrict__ table, bf16* __restrict__ out, int H, int rank,
                             const void* __restrict__ sinks, int sink_dtype) {
    gi_pdl_start();
    __shared__ float w_s[LC_THREADS];
    __shared__ float red[2];
    const int t = blockIdx.x, h = blockIdx.y, lane = threadIdx.x & 31, c0 = 2 * (blockIdx.z * LC_THREADS * NP + threadIdx.x);
    const size_t stride = (size_t)rank + 2, step = (size_t)H * stride;
    const int2 mine = table[t];
    const float* base = part + ((size_t)mine.x * H + h) * stride;
    const float sink = sinks ? load_w(sinks, sink_dtype, h) : -INFINITY;
    // the maximum and the sum, by a warp; then LC_THREADS slices' weights at a time
    if (threadIdx.x < 32) {
        float M = sink;
        for (int s = lane; s < mine.y; s += 32) M = fmaxf(M, base[s * step]);
        M = warp_max(M);
        float L = 0.f;
        for (int s = lane; s < mine.y; s += 32)
            if (base[s * step] != -INFINITY) L += expf(base[s * step] - M) * base[s * step + 1];
        L = warp_sum(L);
        if (lane == 0) { red[0] = M; red[1] = L + (sinks ? expf(sink - M) : 0.f); }
    }
    __syncthreads();
    const float M = red[0], inv = red[1] > 0.f ? 1.f / red[1] : 0.f;
    float v[2 * NP];
#pragma unroll
    for (int i = 0; i < 2 * NP; ++i) v[i] = 0.f;
    for (int s0 = 0; s0 < mine.y; s0 += LC_THREADS) {
        const int n = min(LC_THREADS, mine.y - s0);
        __syncthreads();
        if ((int)threadIdx.x < n) {
            const float m = base[(s0 + threadIdx.x) * step];
            w_s[threadIdx.x] = m == -INFINITY ? -1.f : expf(m - M);      // -1: a slice in which no score was above minus infinity is left out
        }
        __syncthreads();
        const float* x = base + s0 * step + 2 + c0;
        if (rank % 2 == 0) {                                 // rows of an even number of floats: pairs lie on 8 bytes
#pragma unroll (NP == 1 ? 16 : 4)
            for (int s = 0; s < n; ++s)
#pragma unroll
                for (int p = 0; p < NP; ++p) {
                    const float2 y = c0 + 2 * LC_THREADS * p < rank ? *reinterpret_cast<const float2*>(x + s * step + 2 * LC_THREADS * p) : make_float2(0.f, 0.f);
                    if (!(w_s[s] < 0.f)) {
                        v[2 * p] = fmaf(w_s[s], y.x, v[2 * p]);
                        v[2 * p + 1] = fmaf(w_s[s], y.y, v[2 * p + 1]);
                    }
                }
        } else {
            for (int s = 0; s < n; ++s)
#pragma unroll
                for (int p = 0; p < NP; ++p) {
                    const int c = c0 + 2 * LC_THREADS * p;
                    if (w_s[s] < 0.f) continue;
                    if (c < rank) v[2 * p] = fmaf(w_s[s], x[s * step + 2 * LC_THREADS * p], v[2 * p]);
                    if (c + 1 < rank) v[2 * p + 1] = fmaf(w_s[s], x[s * step + 2 * LC_THREADS * p + 1], v[2 * p + 1]);
                }
        }
    }
    bf16* dst = out + ((size_t)t * H + h) * rank;
#pragma unroll
    for (int p = 0; p < NP; ++p) {
        const int c = c0 + 2 * LC_THREADS * p;
        if (c < rank) dst[c] = __float2bfloat16_rn(v[2 * p] * inv);
        if (c + 1 < rank) dst[c + 1] = __float2bfloat16_rn(v[2 * p + 1] * inv);
    }
}
// A head's columns to one block, or to four where the heads are few.
static int launch_latent_combine(const float* part, const int2* table, void* out, int n_tokens, int H, int rank, const void* sinks,
                                 int sink_dtype, cudaStream_t s) {
    if ((long long)n_tokens * H < 512)
        gi_launch(latent_decode_combine_kernel<1>, dim3(n_tokens, H, (rank + 2 * LC_THREADS - 1) / (2 * LC_THREADS)), dim3(LC_THREADS), 0, s, part,
                  table, (bf16*)out, H, rank, sinks, sink_dtype);
    else
        gi_launch(latent_decode_combine_kernel<2>, dim3(n_tokens, H, (rank + 4 * LC_THREADS - 1) / (4 * LC_THREADS)), dim3(LC_THREADS), 0, s, part,
                  table, (bf16*)out, H, rank, sinks, sink_dtype);
    return gi_check_launch("gi_latent_decode_combine");
}

// part: n_tokens n_splits H (2 + rank) floats (an even number of them), then two ints a token; n_tokens n_splits is the number of blocks (for every 32 heads).
extern "C" int gi_latent_decode(const void* q, const void* pool, const int* block_table, const int* tok_pos,
                                const int* tok_slot, float* part, void* out, int n_tokens, int H, int dk, int rank,
                                int page_size, int max_pages, int n_pool_pages, int n_splits, float scale,
                                const void* sinks, int sink_dtype, int* status, int window, void* stream) {
    GI_REQUIRE(window >= 0, "gi_latent_decode: window %d", window);
    GI_REQUIRE(n_tokens >= 0 && H > 0 && dk > 0 && dk % 8 == 0 && rank > 0 && rank <= dk && rank <= 512,
               "gi_latent_decode: rows of %d (a multiple of 8) with %d value columns (at most 512)", dk, rank);
    GI_REQUIRE(n_splits >= 1 && n_splits <= 64 && H <= 65535 && n_tokens <= 65535, "gi_latent_decode: slices, heads, tokens");
    if (n_tokens == 0) return 0;
    int n_blocks = n_tokens * n_splits, least = 1;
    const int2* table = ld_table(part, (size_t)n_blocks * H * (rank + 2));
    GI_REQUIRE((uintptr_t)part % 8 == 0, "gi_latent_decode: the work space must start on 8 bytes");
    cudaStream_t s = (cudaStream_t)stream;
    {   // tensor cores: rows staged with 4 words of padding past a multiple of 32 words
        const int words16 = ((dk + 15) / 16) * 8;
        const int kw = words16 + ((4 - words16 % 32) + 32) % 32;
        const size_t smem_mma = ((size_t)(32 + LD_KEYS) * kw + 32 * 33 + 32 * 20 + 32) * 4;
        const int n_tiles = (rank + 7) / 8;
        const int NTW = n_tiles > 32 ? 8 : (n_tiles > 16 ? 4 : (n_tiles > 8 ? 2 : 1));
        const size_t smem_q = ((size_t)LW_STAGES * LD_KEYS * kw + 4 * 32 * LW_SLD + 32 * 20 + 32) * 4;
        if (dk <= 576) {
            // as many blocks as the chip holds at once, or two a token where those are more.  Tokens that fill it by themselves are cut
            // into slices of 16 chunks at least: shorter ones cost more blocks than they even out.
            int n_sm = 148, dev = 0;
            if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev);
            const int groups = (H + 31) / 32, at_once = n_sm * LW_PER_SM(dk <= 192 ? 3 : 9) / groups, most = at_once > 2 * n_tokens ? at_once : 2 * n_tokens;
            if (n_blocks > most) n_blocks = most;
            if (n_tokens >= at_once) least = 16;
            table = ld_table(part, (size_t)n_blocks * H * (rank + 2));
#define LDQ_CASE(Q, N)                                                                                                 \
            if ((dk <= 192 ? 3 : 9) == Q && NTW == N) {                                                                \
                if (int rc = gi_reserve_smem((const void*)latent_decode_quarters_kernel<Q, N>, smem_q, "gi_latent_decode")) return rc; \
                gi_launch(latent_decode_quarters_kernel<Q, N>, dim3(n_blocks, groups), dim3(LD_WARPS * 32), smem_q, s, (const bf16*)q, \
                          (const bf16*)pool, block_table, tok_pos, tok_slot, part, H, dk, rank, kw, page_size, max_pages, \
                          n_pool_pages, n_blocks, n_tokens, least, scale, status, window);                                    \
            }
            LDQ_CASE(3, 1) LDQ_CASE(3, 2) LDQ_CASE(3, 4) LDQ_CASE(9, 1) LDQ_CASE(9, 2) LDQ_CASE(9, 4) LDQ_CASE(9, 8)
#undef LDQ_CASE
            int rc = gi_check_launch("gi_latent_decode");
            if (rc) return rc;
            return launch_latent_combine(part, table, out, n_tokens, H, rank, sinks, sink_dtype, s);
        }
        if (smem_mma <= 200 * 1024) {
            dim3 grid_mma(n_blocks, (H + 31) / 32);
#define LDM_CASE(N)                                                                                                    \
            if (NTW == N) {                                                                                            \
                int rc = gi_reserve_smem((const void*)latent_decode_mma_kernel<N>, smem_mma, "gi_latent_decode");      \
                if (rc) return rc;                                                                                     \
                gi_launch(latent_decode_mma_kernel<N>, grid_mma, dim3(LD_WARPS * 32), smem_mma, s, (const bf16*)q,     \
                          (const bf16*)pool, block_table, tok_pos, tok_slot, part, H, dk, rank, kw, page_size, max_pages, \
                          n_pool_pages, n_blocks, n_tokens, least, scale, status, window);                                                      \
            }
            LDM_CASE(1) LDM_CASE(2) LDM_CASE(4) LDM_CASE(8)
#undef LDM_CASE
            int rc = gi_check_launch("gi_latent_decode");
            if (rc) return rc;
            return launch_latent_combine(part, table, out, n_tokens, H, rank, sinks, sink_dtype, s);
        }
    }
    const int HPW = H > 16 ? 4 : (H > 8 ? 2 : 1);
    const int HG = HPW * LD_WARPS;
    const int DPL2 = rank > 256 ? 8 : (rank > 128 ? 4 : (rank > 64 ? 2 : 1));
    const size_t smem = (size_t)HG * dk * 4 + (size_t)LD_KEYS * (dk / 2 + 1) * 4;
    GI_REQUIRE(smem <= 220 * 1024, "gi_latent_decode: rows of %d need %zu bytes of shared memory", dk, smem);
    dim3 grid(n_blocks, (H + HG - 1) / HG);
#define LD_CASE(A, B)                                                                                             \
    if (HPW == A && DPL2 == B) {                                                                                  \
        int rc = gi_reserve_smem((const void*)latent_decode_kernel<A, B>, smem, "gi_latent_decode");              \
        if (rc) return rc;                                                                                        \
        gi_launch(latent_decode_kernel<A, B>, grid, dim3(LD_WARPS * 32), smem, s, (const bf16*)q, (const bf16*)pool, \
                  block_table, tok_pos, tok_slot, part, H, dk, rank, page_size, max_pages, n_pool_pages, n_blocks, \
                  n_tokens, least, scale, status, window);                                                                                 \
    }
    LD_CASE(1, 1) LD_CASE(1, 2) LD_CASE(1, 4) LD_CASE(1, 8)
    LD_CASE(2, 1) LD_CASE(2, 2) LD_CASE(2, 4) LD_CASE(2, 8)
    LD_CASE(4, 1) LD_CASE(4, 2) LD_CASE(4, 4) LD_CASE(4, 8)
#undef LD_CASE
    int rc = gi_check_launch("gi_latent_decode");
    if (rc) return rc;
    return launch_latent_combine(part, table, out, n_tokens, H, rank, sinks, sink_dtype, s);
}
