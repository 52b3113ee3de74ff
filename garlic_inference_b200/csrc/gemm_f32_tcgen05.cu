// True float32 matrix product for the 32-bit engine on tensor cores: C[M,N] = A[M,K] . W[N,K]^T for weights of a million elements
// and more (gemm_f32.cu has the others).  Upstream has no 32-bit path.
//
// 2^24 times a float32 number is the exact sum of three bfloat16 numbers (gf_split), and products of those are exact in float32.  Of the nine
// products of two such sums the six largest are made (what is left out is at most 2^-25 of a product, below its rounding to
// float32).  The accumulator starts from zero for every 64 inputs, takes the five small products of all of them first and the
// large one last, and these sums meet in registers by float32 adds that round to nearest, in ascending order: the tensor
// core cuts its own sums off, which is why they are kept that short.  Relative error (2-norm) against 64 bits in units of
// 1e-8, FMAs in order / this, normal inputs: K 256 29 / 8.7, 1,024 57 / 11, 2,048 81 / 13, 5,632 134 / 19, 17,408 237 / 31; the largest
// error of one output in units of |a| |w|: 2.8e-7 / 6.6e-8.
//
// 128 rows of W are the wide side of the tensor core and NT rows of A the other, whatever M is, and an output's products and
// adds do not depend on NT or on the other rows: a row's bits are the same in a prompt, in a decode step and in a batch.
//   warps 0..7     split W: TMA brings 128 x 64 floats; a lane takes a row, splits it and puts the three parts into tensor memory,
//                  where the tensor core reads its wide operand from (the two groups of four warps take turns)
//   warps 8..15    add the sums of 64 inputs up and write the outputs (two groups of four, half of the columns each)
//   warp 16, 17    TMA: slices of W, slices of the three parts of A (made by split_rows_kernel before, 6 bytes an element; of few
//                  rows by this warp itself)
//   warp 18, 19    products, a slice each in turn
// Many tiles: a block walks them, all blocks at once a few tiles of W.  Few: the inputs of a tile are shared out among blocks, which
// leave the sums of 64 inputs in memory, and add_sums_kernel adds them in the same order.
#include "tcgen05.cuh"
#include <math.h>

#define GF_BK 64                     // inputs to a slice and to a sum: 2 x 128 bytes of W, 128 of a part of A
#define GF_ROWS 128
#define GF_W_BYTES (GF_ROWS * GF_BK * 4)
#define GF_SPLITTERS 8
#define GF_ADDERS 8
#define GF_THREADS ((GF_SPLITTERS + GF_ADDERS + 4) * 32)
#define GF_A_COLS 96                 // columns of tensor memory of a split slice: 3 parts x 64 inputs in pairs
#define GF_TMEM_COLS 512
#define GF_RING 8                    // slices that may be under way, at most
#define GF_FEW 16                    // up to so many rows are split by the kernel itself

#define GF_ERR_COPY 71
#define GF_ERR_SPLIT 72
#define GF_ERR_MMA 73
#define GF_ERR_ADD 74

struct GfControl {
    unsigned long long w_full[GF_RING], w_empty[GF_RING], a_full[GF_RING], split[GF_RING], done[GF_RING], acc_full[4], acc_empty[4];
    unsigned int tmem_base;
    int abort;
};

template <int NT> struct GfShape {
    static constexpr int PART = NT * GF_BK * 2;                                   // bytes of one part of A in a slice
    // slices of W and of A's parts in shared memory: W's are let go once they are split, A's after their products
    static constexpr int WS = NT == 128 ? 2 : NT == 16 ? 5 : NT == 96 ? 3 : 4, AS = NT == 128 || NT == 96 ? 3 : NT == 64 ? 4 : NT == 32 ? 6 : 8;
    static constexpr int ACCS = NT <= 32 ? 4 : NT <= 96 ? 3 : 2, SPLITS = NT <= 32 ? 4 : NT == 64 ? 3 : 2;      // accumulators and split slices in tensor memory
    static_assert(WS <= GF_RING && AS <= GF_RING && SPLITS <= GF_RING, "rings");
    static_assert(ACCS * NT + SPLITS * GF_A_COLS <= GF_TMEM_COLS, "tensor memory");
    static constexpr int BYTES = WS * GF_W_BYTES + AS * 3 * PART;
    static constexpr size_t SMEM = (size_t)BYTES + sizeof(GfControl) + 1024;
    static_assert(SMEM <= 232448, "shared memory");
};

// The parts of 2^24 x: of x itself the third would fall under bfloat16's smallest number from 2^-110 down (and the second from 2^-118 down), so
// every float32 number, subnormal ones too, is the exact sum of its parts.  A sum is 2^48 times the output; one that passes the largest
// number with that (an output of 2^80 and more, or an input of 2^104) is not finite and made by FMAs.
#define GF_SCALE 16777216.f
#define GF_UNSCALE (1.f / (GF_SCALE * GF_SCALE))
__device__ __forceinline__ void gf_split(float x, float y, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
    t5_apart(t5_mul2(t5_pair(x, y), t5_pair(GF_SCALE, GF_SCALE)), x, y);
    t5_split3(x, y, hi, mid, lo);
}

__device__ __forceinline__ bool gf_finite(float v) { return fabsf(v) <= 3.402823466e38f; }
// An output whose sum is not finite (the parts of an infinity, and of a number that rounds up to one, are none), by float32 FMAs in order.  K
// is a multiple of 4 and w starts on 16 bytes; 16 words of w are under way at a time.  In us, W of 2,048 x 2,048, one row of A with an
// infinity / all: 300 rows 80 / 1,385 (a float at a time, in front of the stores, 212 / 9,121), 1 row 165 (569), 8 521 / 714 (1,381 / 2,059); finite
// 34, 14 and 15.
__device__ __noinline__ float gf_plain(const float* a, const float* w, int K) {
    float s = 0.f;
#pragma unroll 1
    for (int k0 = 0; k0 < K; k0 += 64) {
        float4 x[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) x[i] = *reinterpret_cast<const float4*>(w + min(k0 + 4 * i, K - 4));
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const float* y = a + k0 + 4 * i;
            if (k0 + 4 * i < K) { s = fmaf(y[0], x[i].x, s); s = fmaf(y[1], x[i].y, s); s = fmaf(y[2], x[i].z, s); s = fmaf(y[3], x[i].w, s); }
        }
    }
    return s;
}
// The same for eight rows of A, which a word of w is fetched once for: where many outputs are not finite.
struct GfEight { float v[8]; };
__device__ __noinline__ GfEight gf_eight(const float* a, long long lda, int rows, const float* w, int K) {
    GfEight s;
    const float* of[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) { s.v[j] = 0.f; of[j] = a + (long long)min(j, rows - 1) * lda; }
#pragma unroll 2
    for (int k = 0; k < K; k += 4) {
        const float4 x = *reinterpret_cast<const float4*>(w + k);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const float* y = of[j] + k;
            s.v[j] = fmaf(y[0], x.x, s.v[j]); s.v[j] = fmaf(y[1], x.y, s.v[j]); s.v[j] = fmaf(y[2], x.z, s.v[j]); s.v[j] = fmaf(y[3], x.w, s.v[j]);
        }
    }
    return s;
}

// sums: nothing, or where the sums of 64 inputs go ([sum][M][N]) when `shares` blocks share the inputs of a tile.
template <int NT>
__global__ void __launch_bounds__(GF_THREADS, 1)
sgemm_split_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_a, const float* __restrict__ A,
                   const float* __restrict__ W, float* __restrict__ C, float* __restrict__ sums, int shares, int M, int N, int K,
                   long long lda, long long ldc, int* __restrict__ error_flag) {
    using S = GfShape<NT>;
    gi_pdl_launch_dependents();
    extern __shared__ unsigned char gf_raw[];
    unsigned char* smem = (unsigned char*)(((uintptr_t)gf_raw + 1023) & ~(uintptr_t)1023);
    GfControl* ctl = reinterpret_cast<GfControl*>(smem + S::BYTES);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int m_tiles = (M + NT - 1) / NT, tiles = m_tiles * ((N + GF_ROWS - 1) / GF_ROWS);
    // this block's tiles are t0, t0 + step, ..., of each the sums u0 .. u1 - 1
    const int all = (K + GF_BK - 1) / GF_BK, share = blockIdx.x % shares;
    const int t0 = blockIdx.x / shares, step = gridDim.x / shares, u0 = (int)((long long)all * share / shares), u1 = (int)((long long)all * (share + 1) / shares);
    const int n_sums = u1 - u0, own = (t0 < tiles ? (tiles - 1 - t0) / step + 1 : 0) * n_sums;      // slices of all of them
    volatile int* abort = &ctl->abort;

    if (threadIdx.x == 0) {
        for (int s = 0; s < GF_RING; ++s) {
            t5_bar_init(&ctl->w_full[s], 1); t5_bar_init(&ctl->w_empty[s], 4); t5_bar_init(&ctl->a_full[s], 1);
            t5_bar_init(&ctl->split[s], 4); t5_bar_init(&ctl->done[s], 1);
        }
        for (int s = 0; s < 4; ++s) { t5_bar_init(&ctl->acc_full[s], 1); t5_bar_init(&ctl->acc_empty[s], GF_ADDERS); }
        ctl->abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 19) t5_alloc(&ctl->tmem_base, GF_TMEM_COLS);
    t5_fence_before();
    __syncthreads();
    t5_fence_after();
    const uint32_t tmem = ctl->tmem_base, split0 = tmem + S::ACCS * NT;

    if (warp < GF_SPLITTERS) {
        gi_pdl_wait();
        const int q = warp & 3, row = q * 32 + lane, swap = row & 7;
        for (int it = warp >> 2; it < own; it += 2) {
            const int s = it % S::WS, last = it - S::SPLITS;                    // the slice that had these columns before
            const uint32_t at = split0 + it % S::SPLITS * GF_A_COLS + ((uint32_t)(q * 32) << 16);
            // In a ring of odd length the slice before this one in its place is the other group's, and may not even have landed: the barrier
            // would then be a phase behind, and its parity say that this slice is there.  So first wait until that one has been let go.
            if (S::WS % 2 && it >= S::WS && !t5_warp_wait(&ctl->w_empty[s], (it / S::WS & 1) ^ 1, abort, error_flag, GF_ERR_SPLIT)) break;
            if (!t5_warp_wait(&ctl->w_full[s], it / S::WS & 1, abort, error_flag, GF_ERR_SPLIT)) break;
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const unsigned char* src = smem + s * GF_W_BYTES + half * (GF_W_BYTES / 2) + row * 128;
                uint32_t part[3][16];
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    const float4 v = *reinterpret_cast<const float4*>(src + ((c ^ swap) << 4));      // as the 128-byte swizzle put them
                    gf_split(v.x, v.y, part[0][2 * c], part[1][2 * c], part[2][2 * c]);
                    gf_split(v.z, v.w, part[0][2 * c + 1], part[1][2 * c + 1], part[2][2 * c + 1]);
                }
                if (half == 0) {
                    if (last >= 0 && !t5_warp_wait(&ctl->done[last % GF_RING], last / GF_RING & 1, abort, error_flag, GF_ERR_SPLIT)) { it = own; break; }
                    t5_fence_after();
                } else {
                    __syncwarp();
                    if (lane == 0) t5_bar_arrive(&ctl->w_empty[s]);
                }
#pragma unroll
                for (int p = 0; p < 3; ++p) t5_st16(at + p * 32 + half * 16, part[p]);
            }
            t5_wait_st();
            t5_fence_before();
            __syncwarp();
            if (lane == 0) t5_bar_arrive(&ctl->split[it % GF_RING]);
        }
    } else if (warp < GF_SPLITTERS + GF_ADDERS) {
        gi_pdl_wait();
        constexpr int COLS = NT / 2, LD = COLS % 16 ? 8 : 16;
        const int q = warp & 3, group = (warp - GF_SPLITTERS) >> 2;
        const uint32_t at = tmem + ((uint32_t)(q * 32) << 16) + group * COLS;
        int it = 0;                      // sums so far
        bool ok = true;
        for (int t = t0; t < tiles && ok; t += step) {
            const int n = t / m_tiles * GF_ROWS + q * 32 + lane, m0 = t % m_tiles * NT + group * COLS;
            t5_f2 sum[COLS / 2];
#pragma unroll
            for (int c = 0; c < COLS / 2; ++c) sum[c] = 0ull;
            for (int u = u0; u < u1; ++u, ++it) {
                const int b = it % S::ACCS;
                if (!t5_warp_wait(&ctl->acc_full[b], it / S::ACCS & 1, abort, error_flag, GF_ERR_ADD)) { ok = false; break; }
                t5_fence_after();
#pragma unroll
                for (int c = 0; c < COLS; c += LD) {
                    float r[LD];
                    t5_ld<LD>(at + b * NT + c, r);
                    t5_wait_ld();
#pragma unroll
                    for (int i = 0; i < LD; i += 2) {
                        const t5_f2 v = t5_pair(r[i], r[i + 1]);
                        sum[(c + i) / 2] = sums ? v : t5_add2(sum[(c + i) / 2], v);
                    }
                }
                t5_fence_before();
                __syncwarp();
                if (lane == 0) t5_bar_arrive(&ctl->acc_empty[b]);
                if (sums && n < N)
#pragma unroll
                    for (int c = 0; c < COLS; ++c)
                        if (m0 + c < M) {
                            float pair[2];
                            t5_apart(sum[c / 2], pair[0], pair[1]);
                            sums[((size_t)u * M + m0 + c) * N + n] = pair[c % 2];
                        }
            }
            if (!ok || sums) continue;
            bool finite = true;
#pragma unroll
            for (int c = 0; c < COLS; ++c)
                if (n < N && m0 + c < M) {
                    float pair[2];
                    t5_apart(sum[c / 2], pair[0], pair[1]);
                    finite = finite && gf_finite(pair[c % 2]);
                    C[(size_t)(m0 + c) * ldc + n] = pair[c % 2] * GF_UNSCALE;
                }
            if (!__all_sync(0xffffffffu, finite))            // (what is not finite is so in C too)
                for (int c0 = 0; c0 < min(COLS, M - m0); c0 += 8) {
                    const int rows = min(8, M - m0 - c0), of = min(n, N - 1);
                    unsigned mine = 0;                       // this lane's outputs that are not finite
                    int columns = 0;
                    for (int c = 0; c < rows; ++c) {
                        const bool odd = n < N && !gf_finite(C[(size_t)(m0 + c0 + c) * ldc + of]);
                        mine |= (unsigned)odd << c;
                        columns += __any_sync(0xffffffffu, odd);
                    }
                    const float *a = A + (size_t)(m0 + c0) * lda, *w = W + (size_t)of * K;
                    if (columns > 2) {
                        const GfEight v = gf_eight(a, lda, rows, w, K);
#pragma unroll
                        for (int c = 0; c < 8; ++c)
                            if (mine >> c & 1) C[(size_t)(m0 + c0 + c) * ldc + n] = v.v[c];
                    } else {
                        for (int c = 0; c < rows; ++c)
                            if (mine >> c & 1) C[(size_t)(m0 + c0 + c) * ldc + n] = gf_plain(a + c * lda, w, K);
                    }
                }
        }
    } else if (NT == GF_FEW && warp == 17) {
        // few rows: this warp makes their parts itself, which saves a launch.  Two lanes to a row, 32 inputs each, a slice ahead.
        gi_pdl_wait();
        const int r = lane >> 1, k_of = (lane & 1) * 32;
        const bool vec = lda % 4 == 0 && (uintptr_t)A % 16 == 0;
        int t = t0, k = u0 * GF_BK;
        float4 v[8];
        auto fetch = [&]() {
            const int m = t % m_tiles * NT + r;
            const float* src = A + (size_t)min(m, M - 1) * lda;
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                const int at = k + k_of + 4 * c;             // K is a multiple of 4
                v[c] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (m < M && at < K) {
                    if (vec) v[c] = *reinterpret_cast<const float4*>(src + at);
                    else v[c] = make_float4(src[at], src[at + 1], src[at + 2], src[at + 3]);
                }
            }
            if ((k += GF_BK) == u1 * GF_BK) {
                k = u0 * GF_BK;
                t += step;
            }
        };
        if (own > 0) fetch();
        for (int it = 0; it < own; ++it) {
            const int s = it % S::AS, last = it - S::AS;
            uint32_t part[3][16];
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                gf_split(v[c].x, v[c].y, part[0][2 * c], part[1][2 * c], part[2][2 * c]);
                gf_split(v[c].z, v[c].w, part[0][2 * c + 1], part[1][2 * c + 1], part[2][2 * c + 1]);
            }
            if (it + 1 < own) fetch();
            if (last >= 0 && !t5_warp_wait(&ctl->done[last % GF_RING], last / GF_RING & 1, abort, error_flag, GF_ERR_COPY)) break;
            unsigned char* row = smem + S::WS * GF_W_BYTES + s * 3 * S::PART + r * 128;
#pragma unroll
            for (int p = 0; p < 3; ++p)
#pragma unroll
                for (int c = 0; c < 4; ++c)                  // 8 inputs, where the 128-byte swizzle wants them
                    *reinterpret_cast<uint4*>(row + p * S::PART + ((((lane & 1) * 4 + c) ^ (r & 7)) << 4)) =
                        make_uint4(part[p][4 * c], part[p][4 * c + 1], part[p][4 * c + 2], part[p][4 * c + 3]);
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) t5_bar_arrive(&ctl->a_full[s]);
        }
    } else if (warp < GF_SPLITTERS + GF_ADDERS + 2) {
        if (lane == 0) {
            // W is nobody's output: its first slices are asked for before the kernel that makes A's parts has finished
            const bool of_w = warp == 16;
            if (!of_w) gi_pdl_wait();
            int t = t0, k = u0 * GF_BK, armed = 0, y = of_w ? t / m_tiles * GF_ROWS : t % m_tiles * NT;
            const int ring = of_w ? S::WS : S::AS;
            for (int it = 0, s = 0, turn = 0; it < own; ++it) {
                const int last = it - S::AS;
                if (of_w ? turn > 0 && !t5_lane_wait(&ctl->w_empty[s], (turn & 1) ^ 1, abort, error_flag, GF_ERR_COPY)
                         : last >= 0 && !t5_lane_wait(&ctl->done[last % GF_RING], last / GF_RING & 1, abort, error_flag, GF_ERR_COPY)) break;
                if (of_w) {
                    t5_bar_expect(&ctl->w_full[s], GF_W_BYTES);
                    t5_load_2d(smem + s * GF_W_BYTES, &map_w, k, y, &ctl->w_full[s]);
                    t5_load_2d(smem + s * GF_W_BYTES + GF_W_BYTES / 2, &map_w, k + GF_BK / 2, y, &ctl->w_full[s]);
                } else {
                    t5_bar_expect(&ctl->a_full[s], 3 * S::PART);
                    t5_load_3d(smem + S::WS * GF_W_BYTES + s * 3 * S::PART, &map_a, k, y, 0, &ctl->a_full[s]);
                }
                armed = it + 1;
                if (++s == ring) { s = 0; ++turn; }
                if ((k += GF_BK) == u1 * GF_BK) {
                    k = u0 * GF_BK;
                    t += step;
                    y = of_w ? t / m_tiles * GF_ROWS : t % m_tiles * NT;
                }
            }
            if (of_w) gi_pdl_wait();
            if (*abort) {                                    // the copies still in flight land before the block leaves
                int never = 0;
                for (int i = max(0, armed - ring); i < armed; ++i) t5_bar_wait(of_w ? &ctl->w_full[i % ring] : &ctl->a_full[i % ring], i / ring & 1, &never);
            }
        }
    } else {
        const bool chosen = t5_elect();
        constexpr uint32_t idesc = t5_idesc(GF_ROWS, NT);
        for (int it = warp - 18; it < own; it += 2) {
            const int b = it % S::ACCS;
            if (!t5_warp_wait(&ctl->acc_empty[b], (it / S::ACCS & 1) ^ 1, abort, error_flag, GF_ERR_MMA)) break;
            if (!t5_warp_wait(&ctl->a_full[it % S::AS], it / S::AS & 1, abort, error_flag, GF_ERR_MMA)) break;
            if (!t5_warp_wait(&ctl->split[it % GF_RING], it / GF_RING & 1, abort, error_flag, GF_ERR_MMA)) break;
            t5_fence_after();
            const uint32_t d = tmem + b * NT, w = split0 + it % S::SPLITS * GF_A_COLS;
            const uint64_t x = t5_desc<128>(t5_smem(smem + S::WS * GF_W_BYTES + it % S::AS * 3 * S::PART));
            if (chosen) {
                constexpr int OF_W[6] = {2, 0, 1, 1, 0, 0}, OF_A[6] = {0, 2, 1, 0, 1, 0};
#pragma unroll
                for (int p = 0; p < 6; ++p)
#pragma unroll
                    for (int k = 0; k < GF_BK / 16; ++k)                 // 16 inputs: 8 columns of tensor memory, 32 bytes of a row of A
                        t5_mma_ts(d, w + OF_W[p] * 32 + k * 8, x + (OF_A[p] * S::PART >> 4) + k * 2, idesc, p | k);
                t5_commit(&ctl->done[it % GF_RING]);
                t5_commit(&ctl->acc_full[b]);
            }
            __syncwarp();
        }
    }
    t5_fence_before();
    __syncthreads();
    if (warp == 19) {
        t5_fence_after();
        t5_free(tmem, GF_TMEM_COLS);
    }
}

// C[m, n] = the sums of 64 inputs added in ascending order, as the kernel above does in registers
__global__ void __launch_bounds__(256)
add_sums_kernel(const float* __restrict__ sums, const float* __restrict__ A, const float* __restrict__ W, float* __restrict__ C, int n_sums,
                int M, int N, int K, long long lda, long long ldc) {
    gi_pdl_start();
    const long long total = (long long)M * N;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
        float v = 0.f;
#pragma unroll 8
        for (int u = 0; u < n_sums; ++u) v += sums[u * total + i];
        const long long m = i / N, n = i - m * N;
        C[m * ldc + n] = gf_finite(v) ? v * GF_UNSCALE : gf_plain(A + m * lda, W + n * K, K);
    }
}

// The three parts of every element of A: parts [3][M][Kp] bfloat16, columns K .. Kp - 1 zero.  Two elements to a thread.
__global__ void __launch_bounds__(256)
split_rows_kernel(const float* __restrict__ A, uint32_t* __restrict__ parts, int M, int K, int Kp, long long lda) {
    gi_pdl_start();
    const int pairs = Kp / 2;
    const long long total = (long long)M * pairs;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
        const long long m = i / pairs;
        const int k = (int)(i - m * pairs) * 2;
        const float* a = A + m * lda + k;
        uint32_t hi, mid, lo;
        gf_split(k < K ? a[0] : 0.f, k + 1 < K ? a[1] : 0.f, hi, mid, lo);
        parts[i] = hi;
        parts[total + i] = mid;
        parts[2 * total + i] = lo;
    }
}

// Which form takes the least time, by what was measured: microseconds a slice of 64 inputs by NT (16: the rows are split by one warp
// a block, the others: a launch before), and what further launches cost.  Shares of the inputs where the tiles would leave half
// of the SMs idle: the sums go through memory.
// In us, this file's product / FMAs in order (gemm_f32.cu), rows x N x K: 1 x 1,024 x 1,024 8.5 / 8.7, 1 x 2,048 x 2,048 14 / 18, 1 x 2,048 x 5,632
// 25 / 46, 1 x 11,264 x 2,048 34 / 31, 8 x 11,264 x 2,048 33 / 57, 17 x 2,048 x 2,048 17 / 34, 100 x 6,144 x 1,024 22 / 77, 491 x 1,024 x 1,024 18 / 121,
// 491 x 2,048 x 2,048 36 / 308, 491 x 11,264 x 2,048 124 / 503, 491 x 2,048 x 5,632 82 / 833, 2,048 x 11,264 x 2,048 517 / 1,722.  Rows of A take 0.82 us a
// slice (64) and 1.55 (128) where the products alone, 24 of 128 x 64 or 128 x 16, take 0.39 and 0.78: the hand-overs between the
// four roles bound both.
struct GfPlan { int nt, shares; };
static GfPlan gf_plan(int M, int N, int K, int n_sm) {
    const int all = (K + GF_BK - 1) / GF_BK, n_tiles = (N + GF_ROWS - 1) / GF_ROWS;
    GfPlan best = {0, 0};
    double least = 1e30;
    static const struct { int nt; double slice; } forms[] = {{16, 1.04}, {32, 0.60}, {64, 0.82}, {96, 1.03}, {128, 1.55}};
    for (const auto& f : forms) {
        if (f.nt == GF_FEW && M > GF_FEW) continue;
        const long long tiles = (long long)((M + f.nt - 1) / f.nt) * n_tiles;
        const double rows = f.nt == GF_FEW ? 0.0 : 2.5, whole = rows + (double)((tiles + n_sm - 1) / n_sm) * all * f.slice;
        if (whole < least) { least = whole; best = {f.nt, 1}; }
        if (tiles * 2 > n_sm) continue;
        const int shares = (int)(n_sm / tiles < all ? n_sm / tiles : all);
        const double shared = rows + 4.0 + (all + shares - 1) / shares * f.slice + (double)M * N * all * 8 / 3e6;
        if (shared < least) { least = shared; best = {f.nt, shares}; }
    }
    return best;
}
extern "C" long long gi_sgemm_split_space(int M, int N, int K) {
    int n_sm = 148, dev = 0;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev);
    const long long parts = 6LL * M * ((K + 7) / 8 * 8);
    const GfPlan p = gf_plan(M, N, K, n_sm);
    return (parts + 255) / 256 * 256 + (p.shares > 1 ? 4LL * M * N * ((K + GF_BK - 1) / GF_BK) : 0);
}
// kernels that one product is
extern "C" int gi_sgemm_split_launches(int M, int N, int K) {
    int n_sm = 148, dev = 0;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev);
    const GfPlan p = gf_plan(M, N, K, n_sm);
    return 1 + (p.nt != GF_FEW) + (p.shares > 1);
}

template <int NT>
static int launch_split(const CUtensorMap& map_w, const float* A, const float* W, float* C, const void* parts, float* sums, int shares, int M, int N,
                        int K, int Kp, long long lda, long long ldc, int n_sm, int* error_flag, cudaStream_t s) {
    CUtensorMap map_a = {};
    if (NT != GF_FEW)
        if (int rc = t5_make_map(&map_a, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, parts, M, Kp, Kp * 2LL, NT, GF_BK, CU_TENSOR_MAP_SWIZZLE_128B, "gi_sgemm_split_nt", 3)) return rc;
    const auto kernel = sgemm_split_kernel<NT>;
    if (int rc = gi_reserve_smem((const void*)kernel, GfShape<NT>::SMEM, "gi_sgemm_split_nt")) return rc;
    const int tiles = (M + NT - 1) / NT * ((N + GF_ROWS - 1) / GF_ROWS);
    gi_launch(kernel, dim3(shares > 1 ? tiles * shares : tiles < n_sm ? tiles : n_sm), dim3(GF_THREADS), GfShape<NT>::SMEM, s, map_w, map_a, A, W, C,
              shares > 1 ? sums : nullptr, shares, M, N, K, lda, ldc, error_flag);
    if (int rc = gi_check_launch("gi_sgemm_split_nt")) return rc;
    if (shares > 1) {
        const long long total = (long long)M * N;
        gi_launch(add_sums_kernel, dim3((unsigned)(total / 256 < 148 * 8 ? total / 256 + 1 : 148 * 8)), dim3(256), 0, s, sums, A, W, C,
                  (K + GF_BK - 1) / GF_BK, M, N, K, lda, ldc);
        return gi_check_launch("gi_sgemm_split_nt");
    }
    return 0;
}

// space: gi_sgemm_split_space(M, N, K) bytes of work space. tile, shares: 0, or a form of its own (tests, measurements).
extern "C" int gi_sgemm_split_nt(const float* A, const float* W, float* C, void* space, long long space_bytes, int M, int N, int K, long long lda, long long ldc,
                                 int tile, int shares, int* error_flag, void* stream) {
    GI_REQUIRE(M >= 0 && N > 0 && K > 0, "gi_sgemm_split_nt: sizes must be positive");
    GI_REQUIRE(lda >= K && ldc >= N, "gi_sgemm_split_nt: row strides shorter than the rows");
    GI_REQUIRE(M <= 1 << 20 && N <= 1 << 24, "gi_sgemm_split_nt: %d rows and %d columns in one product", M, N);
    GI_REQUIRE(K % 4 == 0 && (uintptr_t)W % 16 == 0 && (uintptr_t)space % 16 == 0, "gi_sgemm_split_nt: rows of W must start on 16 bytes");
    GI_REQUIRE(error_flag != nullptr, "gi_sgemm_split_nt: an error flag on the device is required");
    if (M == 0) return 0;
    cudaStream_t s = (cudaStream_t)stream;
    int n_sm = 148, dev = 0;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev);
    const int Kp = (K + 7) / 8 * 8, all = (K + GF_BK - 1) / GF_BK;
    const long long part_bytes = (6LL * M * Kp + 255) / 256 * 256;
    GfPlan plan = gf_plan(M, N, K, n_sm);
    if (tile) plan = {tile, shares < 1 ? 1 : shares > all ? all : shares};
    GI_REQUIRE(part_bytes + (plan.shares > 1 ? 4LL * M * N * all : 0) <= space_bytes, "gi_sgemm_split_nt: %lld bytes of work space are too few", space_bytes);
    float* sums = (float*)((char*)space + part_bytes);
    CUtensorMap map_w;
    if (int rc = t5_make_map(&map_w, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, W, N, K, K * 4LL, GF_ROWS, GF_BK / 2, CU_TENSOR_MAP_SWIZZLE_128B, "gi_sgemm_split_nt")) return rc;
    if (plan.nt != GF_FEW) {
        const long long pairs = (long long)M * (Kp / 2);
        gi_launch(split_rows_kernel, dim3((unsigned)(pairs / 256 < 148 * 8 ? pairs / 256 + 1 : 148 * 8)), dim3(256), 0, s, A, (uint32_t*)space, M, K, Kp, lda);
        if (int rc = gi_check_launch("gi_sgemm_split_nt")) return rc;
    }
#define GF_CASE(NT) if (plan.nt == NT) return launch_split<NT>(map_w, A, W, C, space, sums, plan.shares, M, N, K, Kp, lda, ldc, n_sm, error_flag, s)
    GF_CASE(16);
    GF_CASE(32);
    GF_CASE(64);
    GF_CASE(96);
    GF_CASE(128);
#undef GF_CASE
    GI_REQUIRE(false, "gi_sgemm_split_nt: tiles of %d rows", plan.nt);
}
