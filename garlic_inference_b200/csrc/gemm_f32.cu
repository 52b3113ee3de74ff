// True float32 matrix product for the 32-bit engine: C[M,N] = A[M,K] . W[N,K]^T
// with float32 FMA on the CUDA cores, for weights that gemm_f32_tcgen05.cu does
// not take (small ones, and rows that do not start on 16 bytes).  Each output element is one accumulator summed over k in ascending
// order, so a row's result is the same bits whatever M is: whole prompts,
// single tokens and batches agree exactly, and so do the two kernels here.
//
// Upstream multiplies with a library in the checkpoint's type only
// (src/src-cuda/mat-ops/gemm/gemm.cu:22-41, y = x W^T with W [out, in]); it has
// no 32-bit path.
#include "common.cuh"
#include <math.h>

typedef unsigned long long f32x2;            // two floats in a register pair; each half of fma2 is rounded like fmaf
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ f32x2 both2(float x) {
    f32x2 d;
    asm("mov.b64 %0, {%1, %1};" : "=l"(d) : "f"(x));
    return d;
}
__device__ __forceinline__ void apart2(f32x2 v, float& x, float& y) { asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(v)); }

// ---- many rows: tiles of BM x BN outputs, TM x TN of them to a thread as pairs of neighbouring columns.
// Bound by the FMA pipe.  A slice of SG_BK inputs of both operands lies in shared memory transposed ([k][row], so that a
// thread's rows and columns are whole 16-byte words); the next slice is on its way in registers meanwhile and goes to the
// other buffer, and the values of the next k come out of shared memory while this one's are multiplied.  A thread's rows
// and columns come in words of four that lie BM / (TM / 4) and BN / (TN / 4) apart, so that neighbouring threads read
// neighbouring words.
#define SG_BK 16
template <int BM, int BN, int TM, int TN>
__global__ void __launch_bounds__(BM * BN / (TM * TN))
sgemm_tile_kernel(const float* __restrict__ A, const float* __restrict__ W, float* __restrict__ C,
                  int M, int N, int K, long long lda, long long ldc, int vec) {
    gi_pdl_start();
    constexpr int THREADS = BM * BN / (TM * TN), QA = BM * SG_BK / 4 / THREADS, QW = BN * SG_BK / 4 / THREADS;
    static_assert(QA * THREADS * 4 == BM * SG_BK && QW * THREADS * 4 == BN * SG_BK, "a slice is whole words for every thread");
    __shared__ __align__(16) float As[2][SG_BK][BM + 4];
    __shared__ __align__(16) float Ws[2][SG_BK][BN + 4];
    const int tid = threadIdx.x, tx = tid % (BN / TN), ty = tid / (BN / TN);
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    float4 ra[QA], rw[QW];
    auto word = [&](const float* p, int k, bool in) {        // four inputs of one row from column k on, zeros outside
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (!in) return v;
        if (vec) {
            if (k < K) v = *reinterpret_cast<const float4*>(p + k);
        } else {
            if (k < K) v.x = p[k];
            if (k + 1 < K) v.y = p[k + 1];
            if (k + 2 < K) v.z = p[k + 2];
            if (k + 3 < K) v.w = p[k + 3];
        }
        return v;
    };
    auto fetch = [&](int k0) {
#pragma unroll
        for (int i = 0; i < QA; ++i) {
            const int id = tid + THREADS * i, r = m0 + id / (SG_BK / 4);
            ra[i] = word(A + (size_t)min(r, M - 1) * lda, k0 + id % (SG_BK / 4) * 4, r < M);
        }
#pragma unroll
        for (int i = 0; i < QW; ++i) {
            const int id = tid + THREADS * i, r = n0 + id / (SG_BK / 4);
            rw[i] = word(W + (size_t)min(r, N - 1) * K, k0 + id % (SG_BK / 4) * 4, r < N);
        }
    };
    auto stage = [&](int b) {
#pragma unroll
        for (int i = 0; i < QA; ++i) {
            const int id = tid + THREADS * i, r = id / (SG_BK / 4), k = id % (SG_BK / 4) * 4;
            As[b][k][r] = ra[i].x; As[b][k + 1][r] = ra[i].y; As[b][k + 2][r] = ra[i].z; As[b][k + 3][r] = ra[i].w;
        }
#pragma unroll
        for (int i = 0; i < QW; ++i) {
            const int id = tid + THREADS * i, r = id / (SG_BK / 4), k = id % (SG_BK / 4) * 4;
            Ws[b][k][r] = rw[i].x; Ws[b][k + 1][r] = rw[i].y; Ws[b][k + 2][r] = rw[i].z; Ws[b][k + 3][r] = rw[i].w;
        }
    };
    float a[2][TM];
    f32x2 w[2][TN / 2];
    auto operands = [&](int b, int k, int to) {
#pragma unroll
        for (int i = 0; i < TM / 4; ++i)
            *reinterpret_cast<float4*>(a[to] + 4 * i) = *reinterpret_cast<const float4*>(&As[b][k][ty * 4 + i * (BM / (TM / 4))]);
#pragma unroll
        for (int j = 0; j < TN / 4; ++j) {
            const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(&Ws[b][k][tx * 4 + j * (BN / (TN / 4))]);
            w[to][2 * j] = v.x;
            w[to][2 * j + 1] = v.y;
        }
    };
    f32x2 acc[TM][TN / 2];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN / 2; ++j) acc[i][j] = 0ull;
    fetch(0);
    stage(0);
    __syncthreads();
    for (int k0 = 0, b = 0; k0 < K; k0 += SG_BK, b ^= 1) {
        const bool more = k0 + SG_BK < K;
        if (more) fetch(k0 + SG_BK);
        operands(b, 0, 0);
#pragma unroll
        for (int k = 0; k < SG_BK; ++k) {
            if (k + 1 < SG_BK) operands(b, k + 1, (k + 1) & 1);
#pragma unroll
            for (int i = 0; i < TM; ++i) {
                const f32x2 aa = both2(a[k & 1][i]);
#pragma unroll
                for (int j = 0; j < TN / 2; ++j) acc[i][j] = fma2(aa, w[k & 1][j], acc[i][j]);
            }
        }
        if (more) stage(b ^ 1);
        __syncthreads();
    }
    const bool whole = ldc % 4 == 0 && (uintptr_t)C % 16 == 0;
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int gm = m0 + ty * 4 + i / 4 * (BM / (TM / 4)) + i % 4;
        if (gm >= M) continue;
#pragma unroll
        for (int j = 0; j < TN / 4; ++j) {
            const int gn = n0 + tx * 4 + j * (BN / (TN / 4));
            float v[4];
            apart2(acc[i][2 * j], v[0], v[1]);
            apart2(acc[i][2 * j + 1], v[2], v[3]);
            float* dst = C + (size_t)gm * ldc + gn;
            if (whole && gn + 3 < N) *reinterpret_cast<float4*>(dst) = make_float4(v[0], v[1], v[2], v[3]);
            else
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (gn + e < N) dst[e] = v[e];
        }
    }
}

// ---- few rows (decode steps, short prompts): SV_BN columns and MP rows to a block, a column and MT rows to a thread, both
// operands streamed through a ring of SV_STAGES slices of SV_BK inputs by asynchronous copies.  Up to 16 rows it is bound by
// the chain of K dependent additions of an output (4 cycles each: 4.3 us for 2,048), which bit-equality with the
// kernel above asks for.
#define SV_BN 16
#define SV_BK 128
#define SV_LD (SV_BK + 4)            // neighbouring rows start 4 banks apart
#define SV_STAGES 4
template <int MP, int MT, bool VEC>
__global__ void __launch_bounds__(128)
sgemm_rows_kernel(const float* __restrict__ A, const float* __restrict__ W, float* __restrict__ C,
                  int M, int N, int K, long long lda, long long ldc) {
    extern __shared__ __align__(16) float sv_smem[];         // [stage][SV_BN rows of W, then MP rows of A][SV_LD]
    const int tid = threadIdx.x, n0 = blockIdx.x * SV_BN, m0 = blockIdx.y * MP, slices = (K + SV_BK - 1) / SV_BK;
    constexpr int ITEM = VEC ? 4 : 1, PER_ROW = SV_BK / ITEM;      // floats to a copy, copies to a row
    auto fetch = [&](int slice, int r_begin, int r_end) {    // rows of a slice: of W below SV_BN, of A from there on
        if (slice >= slices) return;
        float* dst = sv_smem + (size_t)(slice % SV_STAGES) * (SV_BN + MP) * SV_LD;
        for (int id = r_begin * PER_ROW + tid; id < r_end * PER_ROW; id += 128) {
            const int r = id / PER_ROW, kk = id % PER_ROW * ITEM, k = slice * SV_BK + kk;
            const bool of_w = r < SV_BN, in = k < K && (of_w ? n0 + r < N : m0 + r - SV_BN < M);
            const float* src = of_w ? W + (size_t)(in ? n0 + r : 0) * K : A + (size_t)(in ? m0 + r - SV_BN : 0) * lda;
            const uint32_t s = (uint32_t)__cvta_generic_to_shared(dst + r * SV_LD + kk);
            if (VEC) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(src + (in ? k : 0)), "r"(in ? 16 : 0));
            else asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(s), "l"(src + (in ? k : 0)), "r"(in ? 4 : 0));
        }
    };
    // the first slices of W are asked for before the kernel that makes A has finished
    gi_pdl_launch_dependents();
    for (int s = 0; s < SV_STAGES - 1; ++s) fetch(s, 0, SV_BN);
    gi_pdl_wait();
    for (int s = 0; s < SV_STAGES - 1; ++s) {
        fetch(s, SV_BN, SV_BN + MP);
        asm volatile("cp.async.commit_group;\n" ::);         // (the first group also holds every slice of W so far)
    }
    const int nl = tid % SV_BN, ml = tid / SV_BN * MT;
    const bool works = ml < MP;
    float acc[MT];
#pragma unroll
    for (int i = 0; i < MT; ++i) acc[i] = 0.f;
    for (int s = 0; s < slices; ++s) {
        asm volatile("cp.async.wait_group %0;\n" ::"n"(SV_STAGES - 2));
        __syncthreads();                                     // this slice is there, and the one before it is done with
        fetch(s + SV_STAGES - 1, 0, SV_BN + MP);
        asm volatile("cp.async.commit_group;\n" ::);
        if (!works) continue;
        const float* w = sv_smem + (size_t)(s % SV_STAGES) * (SV_BN + MP) * SV_LD + nl * SV_LD;
        const float* a = sv_smem + (size_t)(s % SV_STAGES) * (SV_BN + MP) * SV_LD + (SV_BN + ml) * SV_LD;
        // the next four inputs come out of shared memory while four are summed
        float4 y = *reinterpret_cast<const float4*>(w), x[MT];
#pragma unroll
        for (int i = 0; i < MT; ++i) x[i] = *reinterpret_cast<const float4*>(a + i * SV_LD);
#pragma unroll 8
        for (int k = 4; k <= SV_BK; k += 4) {                // (the last round reads the rows' padding and drops it)
            const float4 yn = *reinterpret_cast<const float4*>(w + k);
            float4 xn[MT];
#pragma unroll
            for (int i = 0; i < MT; ++i) xn[i] = *reinterpret_cast<const float4*>(a + i * SV_LD + k);
#pragma unroll
            for (int i = 0; i < MT; ++i) acc[i] = fmaf(x[i].x, y.x, acc[i]);
#pragma unroll
            for (int i = 0; i < MT; ++i) acc[i] = fmaf(x[i].y, y.y, acc[i]);
#pragma unroll
            for (int i = 0; i < MT; ++i) acc[i] = fmaf(x[i].z, y.z, acc[i]);
#pragma unroll
            for (int i = 0; i < MT; ++i) acc[i] = fmaf(x[i].w, y.w, acc[i]);
            y = yn;
#pragma unroll
            for (int i = 0; i < MT; ++i) x[i] = xn[i];
        }
    }
    if (!works || n0 + nl >= N) return;
#pragma unroll
    for (int i = 0; i < MT; ++i)
        if (m0 + ml + i < M) C[(size_t)(m0 + ml + i) * ldc + n0 + nl] = acc[i];
}

template <int BM, int BN, int TM, int TN>
static void launch_tiles(const float* A, const float* W, float* C, int M, int N, int K, long long lda, long long ldc, int vec,
                         cudaStream_t s) {
    dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
    gi_launch(sgemm_tile_kernel<BM, BN, TM, TN>, grid, dim3(BM * BN / (TM * TN)), 0, s, A, W, C, M, N, K, lda, ldc, vec);
}
template <int MP, int MT>
static int launch_rows(const float* A, const float* W, float* C, int M, int N, int K, long long lda, long long ldc, int vec,
                       cudaStream_t s) {
    const size_t smem = (size_t)SV_STAGES * (SV_BN + MP) * SV_LD * sizeof(float);
    const auto kernel = vec ? sgemm_rows_kernel<MP, MT, true> : sgemm_rows_kernel<MP, MT, false>;
    if (int rc = gi_reserve_smem((const void*)kernel, smem, "gi_sgemm_nt")) return rc;
    gi_launch(kernel, dim3((N + SV_BN - 1) / SV_BN, (M + MP - 1) / MP), dim3(128), smem, s, A, W, C, M, N, K, lda, ldc);
    return 0;
}

extern "C" int gi_sgemm_nt(const float* A, const float* W, float* C, int M, int N, int K, long long lda,
                           long long ldc, void* stream) {
    GI_REQUIRE(M >= 0 && N > 0 && K > 0, "gi_sgemm_nt: sizes must be positive");
    GI_REQUIRE(lda >= K && ldc >= N, "gi_sgemm_nt: row strides shorter than the rows");
    if (M == 0) return 0;
    GI_REQUIRE(((long long)M + 63) / 64 <= 65535, "gi_sgemm_nt: %d rows in one product is beyond %d", M, 65535 * 64);
    const int vec = K % 4 == 0 && lda % 4 == 0 && ((uintptr_t)A | (uintptr_t)W) % 16 == 0;
    cudaStream_t s = (cudaStream_t)stream;
    // Every kernel and tile gives the same bits, so the choice is by time alone: the least of what each was measured to take
    // per input k when it puts c blocks on the SM that gets most (148 SMs; one block alone waits for shared memory between
    // its products, several fill the pipe).  Whole products, first the 64 x 64 tiles of 4 x 4 a thread that all sizes had
    // before, then what is chosen now, in us:
    //   rows x N x K   1 x 2,048 x 2,048   32 x 11,264 x 2,048   491 x 2,048 x 2,048   491 x 11,264 x 2,048   2,048 x 11,264 x 2,048
    //   before                143                  250                   228                  1,073                   4,056
    //   now                    19                   94                   129                    494                   1,720
    auto blocks = [&](long long bm, long long bn) { return (double)((((M + bm - 1) / bm) * ((N + bn - 1) / bn) + 147) / 148); };
    if (M <= 16) {
        const int rc = M == 1   ? launch_rows<1, 1>(A, W, C, M, N, K, lda, ldc, vec, s)
                       : M <= 4 ? launch_rows<4, 4>(A, W, C, M, N, K, lda, ldc, vec, s)
                       : M <= 8 ? launch_rows<8, 4>(A, W, C, M, N, K, lda, ldc, vec, s)
                                : launch_rows<16, 4>(A, W, C, M, N, K, lda, ldc, vec, s);
        if (rc) return rc;
        return gi_check_launch("gi_sgemm_nt");
    }
    const double c_rows = blocks(32, SV_BN), c32 = blocks(32, 64), c64 = blocks(64, 64), c_b = blocks(64, 128), c_w = blocks(128, 128);
    const double t_rows = c_rows <= 1 ? 15.5 : c_rows <= 2 ? 22.0 : 11.4 * c_rows + 6.0;      // ns a k
    const double t32 = c32 <= 1 ? 32.0 : c32 <= 2 ? 48.0 : 20.0 * c32;
    const double t64 = c64 <= 2 ? 62.0 : 51.0 * ((long long)(c64 + 1) / 2);             // two warps: every second block shares their schedulers
    const double t_b = c_b <= 1 ? 68.0 : 51.0 * c_b, t_w = c_w <= 1 ? 100.0 : 89.0 * c_w;
    // (tiles of 32 rows take half as many rows in one launch as the check above lets through)
    const bool tall = ((long long)M + 31) / 32 > 65535;
    const double least = fmin(tall ? t64 : fmin(t_rows, t32), fmin(t64, fmin(t_b, t_w)));
    if (!tall && least == t_rows) {
        if (int rc = launch_rows<32, 4>(A, W, C, M, N, K, lda, ldc, vec, s)) return rc;
    } else if (!tall && least == t32) launch_tiles<32, 64, 4, 4>(A, W, C, M, N, K, lda, ldc, vec, s);
    else if (least == t64) launch_tiles<64, 64, 8, 8>(A, W, C, M, N, K, lda, ldc, vec, s);
    else if (least == t_b) launch_tiles<64, 128, 8, 8>(A, W, C, M, N, K, lda, ldc, vec, s);
    else launch_tiles<128, 128, 8, 16>(A, W, C, M, N, K, lda, ldc, vec, s);
    return gi_check_launch("gi_sgemm_nt");
}
