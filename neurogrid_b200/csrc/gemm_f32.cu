// True 32-bit matrix product for the float32 path:  C[M,N] = A[M,K] * W[N,K]^T (+ bias[N]).
//
// FFMA only: no tensor cores, no TF32.  The order of the additions depends on K alone: k is cut into chunks of 64; a
// chunk has two sums, of its even and of its odd k, each in ascending order (the two halves of one packed FMA), which
// are added; the chunks' sums are added in ascending order.  Both kernels below form exactly that, so a row's result
// does not depend on M, on the other rows of the batch or on where the row sits in it, and shorter chains of
// additions are a little nearer to 64 bits than one chain over k.  The reference calls cuBLAS for every contraction
// (gpu/cuda/matmul.cu:316-355) and has no float32 path.
//
// Few rows (single tokens) are bound by the weights' bytes: `gemm_f32_rows_kernel`.  More rows are bound by the FMA
// pipe: `gemm_f32_tile_kernel`.  Measured on the 350M LFM2 shape, two prompts of 96 tokens and 8 decode steps, where
// one kernel of 64 x 64 tiles (4 x 4 elements a thread, synchronous loads) took 109 ms of the pass: the products of
// the decode steps now take 3.8 ms (7.4 us each, the weights at 3.0 TB/s), those of the prompts' step of 256 padded
// rows 6.3 ms (gate/up, 256 x 9216 x 1024: 138 us, 35 of 74 TFLOP/s).
#include "ng_common.cuh"

#define GF_CHUNK 64

__device__ __forceinline__ uint64_t gf_fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ float gf_both(uint64_t v) {
    return __uint_as_float((uint32_t)v) + __uint_as_float((uint32_t)(v >> 32));
}
// 16 bytes of shared memory as two pairs of floats
__device__ __forceinline__ ulonglong2 gf_lds(const float* p) { return *reinterpret_cast<const ulonglong2*>(p); }

// Four floats to shared memory, asynchronously; elements from `have` on become zero.  AL: the source is 16-byte
// aligned whenever all four are there; otherwise each element is copied by itself.
template <bool AL>
__device__ __forceinline__ void gf_copy4(float* dst, const float* src, int have) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    if constexpr (AL) {
        const int n = have >= 4 ? 16 : have > 0 ? 4 * have : 0;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
    } else {
#pragma unroll
        for (int i = 0; i < 4; ++i)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d + 4 * i), "l"(i < have ? src + i : src), "r"(i < have ? 4 : 0) : "memory");
    }
}
__device__ __forceinline__ void gf_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void gf_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// ---- few rows --------------------------------------------------------------------------------------------------
// A block owns 8 columns (weight rows) and up to MR rows of A and walks k in pieces of 16 chunks.  A thread owns one
// column and one chunk of the piece for all MR rows; the 16 chunk sums of a (row, column) are then added in order by
// one thread.  Eight columns a block keep 128 blocks busy at N = 1,024; the pieces' copies (33 KB of weights) run
// GR_STAGES deep, and the first weights are requested before the kernel in front has ended.
#define GR_COLS 8
#define GR_CH 16
#define GR_K (GR_CH * GF_CHUNK)
#define GR_WROW (GR_K + 4)                       // 4 mod 32 words: eight columns read 16 bytes each without conflicts
#define GR_XROW (GR_CH * (GF_CHUNK + 4))         // chunks 68 words apart: the four chunks a warp reads lie in other banks
#define GR_STAGES 3

template <int MR, bool AL>
__global__ void __launch_bounds__(GR_COLS* GR_CH)
gemm_f32_rows_kernel(const float* __restrict__ A, const float* __restrict__ W, const float* __restrict__ bias,
                     float* __restrict__ C, int M, int N, int K, int lda, int ldw, int ldc, int stages) {
    extern __shared__ __align__(16) float gr_smem[];
    constexpr int STAGE = GR_COLS * GR_WROW + MR * GR_XROW;
    float* part = gr_smem + (size_t)stages * STAGE;                // [2][chunk][MR * GR_COLS]
    const int tid = threadIdx.x, col = tid % GR_COLS, ch = tid / GR_COLS;
    const int n0 = blockIdx.x * GR_COLS, m0 = blockIdx.y * MR;
    const int pieces = (K + GR_K - 1) / GR_K;
    ng_pdl_trigger();

    auto load_w = [&](int p) {
        float* s = gr_smem + (size_t)(p % stages) * STAGE;
        const int k0 = p * GR_K;
        for (int i = tid; i < GR_COLS * (GR_K / 4); i += GR_COLS * GR_CH) {
            const int r = i / (GR_K / 4), k = (i % (GR_K / 4)) * 4;
            if (k0 + k >= ((K + GF_CHUNK - 1) / GF_CHUNK) * GF_CHUNK) continue;
            const int have = n0 + r < N ? K - (k0 + k) : 0;
            gf_copy4<AL>(s + r * GR_WROW + k, have > 0 ? W + (size_t)(n0 + r) * ldw + k0 + k : W, have);
        }
    };
    auto load_x = [&](int p, const float* a) {
        float* s = gr_smem + (size_t)(p % stages) * STAGE + GR_COLS * GR_WROW;
        const int k0 = p * GR_K;
        for (int i = tid; i < MR * (GR_K / 4); i += GR_COLS * GR_CH) {
            const int r = i / (GR_K / 4), k = (i % (GR_K / 4)) * 4;
            if (k0 + k >= ((K + GF_CHUNK - 1) / GF_CHUNK) * GF_CHUNK) continue;
            const int have = m0 + r < M ? K - (k0 + k) : 0;
            gf_copy4<AL>(s + r * GR_XROW + (k / GF_CHUNK) * (GF_CHUNK + 4) + k % GF_CHUNK,
                         have > 0 ? a + (size_t)(m0 + r) * lda + k0 + k : a, have);
        }
    };
    const int ahead = min(stages, pieces);
    for (int p = 0; p < ahead; ++p) load_w(p);
    ng_pdl_wait();
    const float* a = ng_after_wait(A);
    // group p holds piece p; the weights asked for in front of the wait are all in group 0
    for (int p = 0; p < GR_STAGES; ++p) {
        if (p < ahead) load_x(p, a);
        gf_commit();
    }
    float total = 0.f;
    for (int p = 0; p < pieces; ++p) {
        gf_wait<GR_STAGES - 1>();
        __syncthreads();
        const float* s = gr_smem + (size_t)(p % stages) * STAGE;
        const int chunks = min(GR_CH, (K - p * GR_K + GF_CHUNK - 1) / GF_CHUNK);
        float* pp = part + (p & 1) * GR_CH * MR * GR_COLS;
        if (ch < chunks) {
            uint64_t acc[MR];
#pragma unroll
            for (int r = 0; r < MR; ++r) acc[r] = 0ull;
            const float* w = s + col * GR_WROW + ch * GF_CHUNK;
            const float* x = s + GR_COLS * GR_WROW + ch * (GF_CHUNK + 4);
#pragma unroll 8
            for (int k = 0; k < GF_CHUNK; k += 4) {
                const ulonglong2 wv = gf_lds(w + k);
#pragma unroll
                for (int r = 0; r < MR; ++r) {
                    const ulonglong2 xv = gf_lds(x + r * GR_XROW + k);
                    acc[r] = gf_fma2(xv.y, wv.y, gf_fma2(xv.x, wv.x, acc[r]));
                }
            }
#pragma unroll
            for (int r = 0; r < MR; ++r) pp[(ch * MR + r) * GR_COLS + col] = gf_both(acc[r]);
        }
        __syncthreads();
        if (p + stages < pieces) {                               // the stage just read is free
            load_w(p + stages);
            load_x(p + stages, a);
        }
        gf_commit();
        if (tid < MR * GR_COLS)
            for (int c = 0; c < chunks; ++c) total += pp[c * MR * GR_COLS + tid];
    }
    const int m = m0 + tid / GR_COLS, n = n0 + col;
    if (tid < MR * GR_COLS && m < M && n < N) C[(size_t)m * ldc + n] = total + (bias ? bias[n] : 0.f);
}

// ---- more rows -------------------------------------------------------------------------------------------------
// 128 threads form a BM x BN tile, TM x TN elements each.  A stage holds 32 k of both operands as rows of 36 words:
// a thread reads 16 bytes along k (two pairs for the packed FMA), the eight rows a warp reads lie in other banks.
#define GT_BK 32
#define GT_ROW (GT_BK + 4)
#define GT_STAGES 4

template <int BM, int BN, int TM, int TN, bool AL>
__global__ void __launch_bounds__(128)
gemm_f32_tile_kernel(const float* __restrict__ A, const float* __restrict__ W, const float* __restrict__ bias,
                     float* __restrict__ C, int M, int N, int K, int lda, int ldw, int ldc) {
    extern __shared__ __align__(16) float gt_smem[];
    constexpr int STAGE = (BM + BN) * GT_ROW, TR = BM / TM, TC = BN / TN;
    static_assert(TR * TC == 128 && TR == 8, "a warp covers 8 rows x 4 columns of threads");
    const int tid = threadIdx.x, tr = tid % TR, tc = tid / TR;
    const int n0 = blockIdx.x * BN, m0 = blockIdx.y * BM;
    // the order of the sums has whole chunks: an odd number of stages ends with one of zeros
    const int stages = 2 * ((K + GF_CHUNK - 1) / GF_CHUNK);
    ng_pdl_trigger();

    auto load_w = [&](int t) {
        float* s = gt_smem + (t % GT_STAGES) * STAGE + BM * GT_ROW;
#pragma unroll
        for (int i = tid; i < BN * (GT_BK / 4); i += 128) {
            const int r = i / (GT_BK / 4), k = (i % (GT_BK / 4)) * 4, kk = t * GT_BK + k;
            const int have = n0 + r < N ? K - kk : 0;
            gf_copy4<AL>(s + r * GT_ROW + k, have > 0 ? W + (size_t)(n0 + r) * ldw + kk : W, have);
        }
    };
    auto load_a = [&](int t, const float* a) {
        float* s = gt_smem + (t % GT_STAGES) * STAGE;
#pragma unroll
        for (int i = tid; i < BM * (GT_BK / 4); i += 128) {
            const int r = i / (GT_BK / 4), k = (i % (GT_BK / 4)) * 4, kk = t * GT_BK + k;
            const int have = m0 + r < M ? K - kk : 0;
            gf_copy4<AL>(s + r * GT_ROW + k, have > 0 ? a + (size_t)(m0 + r) * lda + kk : a, have);
        }
    };
    for (int t = 0; t < GT_STAGES - 1 && t < stages; ++t) load_w(t);
    ng_pdl_wait();
    const float* a = ng_after_wait(A);
    for (int t = 0; t < GT_STAGES - 1; ++t) {
        if (t < stages) load_a(t, a);
        gf_commit();
    }
    uint64_t acc[TM][TN];
    float total[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0ull, total[i][j] = 0.f;

    for (int t = 0; t < stages; ++t) {
        gf_wait<GT_STAGES - 2>();
        __syncthreads();
        if (t + GT_STAGES - 1 < stages) {                        // into the stage that was read before this barrier
            load_w(t + GT_STAGES - 1);
            load_a(t + GT_STAGES - 1, a);
        }
        gf_commit();
        const float* as = gt_smem + (t % GT_STAGES) * STAGE + tr * GT_ROW;
        const float* ws = gt_smem + (t % GT_STAGES) * STAGE + (BM + tc) * GT_ROW;
#pragma unroll
        for (int k = 0; k < GT_BK; k += 4) {
            ulonglong2 av[TM];
#pragma unroll
            for (int i = 0; i < TM; ++i) av[i] = gf_lds(as + i * TR * GT_ROW + k);
#pragma unroll
            for (int j = 0; j < TN; ++j) {
                const ulonglong2 wv = gf_lds(ws + j * TC * GT_ROW + k);
#pragma unroll
                for (int i = 0; i < TM; ++i) acc[i][j] = gf_fma2(av[i].y, wv.y, gf_fma2(av[i].x, wv.x, acc[i][j]));
            }
        }
        if (t & 1) {                                             // a chunk's end
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) total[i][j] += gf_both(acc[i][j]), acc[i][j] = 0ull;
        }
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int m = m0 + tr + i * TR;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int n = n0 + tc + j * TC;
            if (n < N) C[(size_t)m * ldc + n] = total[i][j] + (bias ? bias[n] : 0.f);
        }
    }
}

template <int MR, bool AL>
static int gf_rows(const float* A, const float* W, const float* bias, float* C, int M, int N, int K, int lda, int ldw,
                   int ldc, cudaStream_t stream) {
    const int pieces = (K + GR_K - 1) / GR_K, stages = pieces < GR_STAGES ? pieces : GR_STAGES;
    constexpr int STAGE = GR_COLS * GR_WROW + MR * GR_XROW, PART = 2 * GR_CH * MR * GR_COLS;
    static std::atomic<unsigned long long> done{0};
    if (!ng_allow_smem(done, gemm_f32_rows_kernel<MR, AL>, (GR_STAGES * STAGE + PART) * 4)) return NG_LAUNCH_FAILED;
    dim3 grid((N + GR_COLS - 1) / GR_COLS, (M + MR - 1) / MR);
    if (grid.y > 65535) return NG_BAD_SIZE;
    NG_LAUNCH((gemm_f32_rows_kernel<MR, AL>), grid, GR_COLS * GR_CH, (size_t)(stages * STAGE + PART) * 4, stream, A, W,
              bias, C, M, N, K, lda, ldw, ldc, stages);
    return ng_launch_status();
}

template <int BM, int BN, int TM, int TN, bool AL>
static int gf_tile(const float* A, const float* W, const float* bias, float* C, int M, int N, int K, int lda, int ldw,
                   int ldc, cudaStream_t stream) {
    constexpr int BYTES = GT_STAGES * (BM + BN) * GT_ROW * 4;
    static std::atomic<unsigned long long> done{0};
    if (!ng_allow_smem(done, gemm_f32_tile_kernel<BM, BN, TM, TN, AL>, BYTES)) return NG_LAUNCH_FAILED;
    dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
    if (grid.y > 65535) return NG_BAD_SIZE;
    NG_LAUNCH((gemm_f32_tile_kernel<BM, BN, TM, TN, AL>), grid, 128, BYTES, stream, A, W, bias, C, M, N, K, lda, ldw, ldc);
    return ng_launch_status();
}

// Rows up to which the few-rows kernel takes the product: it reads the weights once per 8 rows (from the L2 after the
// first time) with 128 blocks at N = 1,024, where 32-row tiles would leave 32 blocks to walk K alone.
#define GF_ROWS_MAX 32

template <bool AL>
static int gf_dispatch(const float* A, const float* W, const float* bias, float* C, int M, int N, int K, int lda,
                       int ldw, int ldc, cudaStream_t s) {
    if (M <= GF_ROWS_MAX) {
        if (M == 1) return gf_rows<1, AL>(A, W, bias, C, M, N, K, lda, ldw, ldc, s);
        if (M == 2) return gf_rows<2, AL>(A, W, bias, C, M, N, K, lda, ldw, ldc, s);
        if (M <= 4) return gf_rows<4, AL>(A, W, bias, C, M, N, K, lda, ldw, ldc, s);
        return gf_rows<8, AL>(A, W, bias, C, M, N, K, lda, ldw, ldc, s);
    }
    auto blocks = [&](int bm, int bn) { return (long long)((M + bm - 1) / bm) * ((N + bn - 1) / bn); };
    if (blocks(64, 64) >= 2 * 148) return gf_tile<64, 64, 8, 4, AL>(A, W, bias, C, M, N, K, lda, ldw, ldc, s);
    if (blocks(32, 64) >= 148) return gf_tile<32, 64, 4, 4, AL>(A, W, bias, C, M, N, K, lda, ldw, ldc, s);
    return gf_tile<32, 32, 4, 2, AL>(A, W, bias, C, M, N, K, lda, ldw, ldc, s);
}

NG_EXPORT int ng_gemm_f32(const float* A, const float* W, const float* bias, float* C, int M, int N, int K,
                          int lda, int ldw, int ldc, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return NG_OK;
    if (K <= 0 || lda < K || ldw < K || ldc < N) return NG_BAD_SIZE;
    // 16-byte copies need every row to begin on a 16-byte boundary (a last piece of fewer than four floats is asked
    // for by its size); other operands are copied a float at a time
    const bool al = (((uintptr_t)A | (uintptr_t)W) & 15) == 0 && lda % 4 == 0 && ldw % 4 == 0;
    return al ? gf_dispatch<true>(A, W, bias, C, M, N, K, lda, ldw, ldc, stream)
              : gf_dispatch<false>(A, W, bias, C, M, N, K, lda, ldw, ldc, stream);
}
