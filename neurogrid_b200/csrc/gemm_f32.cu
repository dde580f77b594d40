// True 32-bit matrix product for the float32 path:  C[M,N] = A[M,K] * W[N,K]^T (+ bias[N]).
//
// FFMA only: no tensor cores, no TF32.  The order of the additions depends on K alone: k is cut into chunks of 64; a
// chunk has two sums, of its even and of its odd k, each in ascending order (the two halves of one packed FMA), which
// are added; the sums of 16 chunks are added in ascending order to a group's, the groups' sums likewise.  Both kernels
// below form exactly that, so a row's result does not depend on M, on the other rows of the batch or on where the row
// sits in it, and shorter chains of additions are a little nearer to 64 bits than one chain over k.  The groups of a
// long K (2 to 8 of them) are walked by one block, or, where that is the faster (gemm_f32_form.h), they are the blocks of a
// cluster, which add their sums through shared memory in the same order.  The reference calls cuBLAS for every contraction
// (gpu/cuda/matmul.cu:316-355) and has no float32 path.
//
// Few rows (single tokens) are bound by the weights' bytes: `gemm_f32_rows_kernel`.  More rows are bound by the FMA
// pipe: `gemm_f32_tile_kernel`.  Measured on the 350M LFM2 shape, two prompts of 96 tokens and 8 decode steps, where
// one kernel of 64 x 64 tiles (4 x 4 elements a thread, synchronous loads) took 109 ms of the pass: the products of
// the decode steps took 3.8 ms, those of the prompts' step of 256 padded rows 6.3 ms; with the groups of a long K side
// by side and 192 rows the pass takes 10.7 ms instead of 13.0 (192 x 1024 x 4608: 75 us instead of 223; 2 rows: 6.2
// instead of 10.8; 192 x 9216 x 1024: 107 us, 34 of 74 TFLOP/s).
#include "gemm_f32_form.h"
#include "ng_common.cuh"

__device__ __forceinline__ uint32_t gf_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void gf_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// the float at `p` of this block's shared memory, in block `rank` of the cluster
__device__ __forceinline__ float gf_peer(const float* p, int rank) {
    uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
    float v;
    asm volatile("{\n\t.reg .u32 r;\n\tmapa.shared::cluster.u32 r, %1, %2;\n\tld.shared::cluster.f32 %0, [r];\n\t}" : "=f"(v) : "r"(a), "r"(rank) : "memory");
    return v;
}

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
// one thread: a group's sum.  Eight columns a block keep 128 blocks busy at N = 1,024, and a cluster's blocks share the
// pieces of a long K; otherwise the pieces' copies (33 KB of weights) run GR_STAGES deep.  The first weights are
// requested before the kernel in front has ended.
#define GR_CH 16
#define GR_K GF_GROUP                            // a piece is a group
#define GR_WROW (GR_K + 4)                       // 4 mod 32 words: eight columns read 16 bytes each without conflicts
#define GR_XROW (GR_CH * (GF_CHUNK + 4))         // chunks 68 words apart: the four chunks a warp reads lie in other banks
#define GR_STAGES 3

template <int MR, bool AL, bool CLUSTER>
__global__ void __launch_bounds__(GR_COLS* GR_CH)
gemm_f32_rows_kernel(const float* __restrict__ A, const float* __restrict__ W, const float* __restrict__ bias,
                     float* __restrict__ C, int M, int N, int K, int lda, int ldw, int ldc, int stages) {
    extern __shared__ __align__(16) float gr_smem[];
    constexpr int STAGE = GR_COLS * GR_WROW + MR * GR_XROW;
    float* part = gr_smem + (size_t)stages * STAGE;                // [2][chunk][MR * GR_COLS]
    const int tid = threadIdx.x, col = tid % GR_COLS, ch = tid / GR_COLS;
    const int n0 = blockIdx.x * GR_COLS, m0 = blockIdx.y * MR;
    const int rank = CLUSTER ? gf_rank() : 0;                      // (the cluster's blocks are those of blockIdx.z)
    const int pieces = CLUSTER ? 1 : (K + GR_K - 1) / GR_K;        // this block's: in a cluster the one of its rank
    ng_pdl_trigger();

    auto load_w = [&](int p) {
        float* s = gr_smem + (size_t)(p % stages) * STAGE;
        const int k0 = (rank + p) * GR_K;
        for (int i = tid; i < GR_COLS * (GR_K / 4); i += GR_COLS * GR_CH) {
            const int r = i / (GR_K / 4), k = (i % (GR_K / 4)) * 4;
            if (k0 + k >= ((K + GF_CHUNK - 1) / GF_CHUNK) * GF_CHUNK) continue;
            const int have = n0 + r < N ? K - (k0 + k) : 0;
            gf_copy4<AL>(s + r * GR_WROW + k, have > 0 ? W + (size_t)(n0 + r) * ldw + k0 + k : W, have);
        }
    };
    auto load_x = [&](int p, const float* a) {
        float* s = gr_smem + (size_t)(p % stages) * STAGE + GR_COLS * GR_WROW;
        const int k0 = (rank + p) * GR_K;
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
        const int chunks = min(GR_CH, (K - (rank + p) * GR_K + GF_CHUNK - 1) / GF_CHUNK);
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
        if (tid < MR * GR_COLS) {
            float group = 0.f;
            for (int c = 0; c < chunks; ++c) group += pp[c * MR * GR_COLS + tid];
            total += group;
        }
    }
    if constexpr (CLUSTER) {
        if (tid < MR * GR_COLS) part[GR_CH * MR * GR_COLS + tid] = total;        // (the half that was not used)
        gf_cluster_sync();
        if (rank == 0 && tid < MR * GR_COLS) {
            total = 0.f;
            for (int r = 0; r < (int)gridDim.z; ++r) total += gf_peer(part + GR_CH * MR * GR_COLS + tid, r);
        }
        gf_cluster_sync();                                       // a block's shared memory is there until it has been read
        if (rank != 0) return;
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

// GROUPS: K is one group (0), the groups of this block's walk one after the other (1), or the blocks of a cluster (2).
template <int BM, int BN, int TM, int TN, bool AL, int GROUPS>
__global__ void __launch_bounds__(128)
gemm_f32_tile_kernel(const float* __restrict__ A, const float* __restrict__ W, const float* __restrict__ bias,
                     float* __restrict__ C, int M, int N, int K, int lda, int ldw, int ldc) {
    extern __shared__ __align__(16) float gt_smem[];
    constexpr int STAGE = (BM + BN) * GT_ROW, TR = BM / TM, TC = BN / TN;
    static_assert(TR * TC == 128 && TR == 8, "a warp covers 8 rows x 4 columns of threads");
    const int tid = threadIdx.x, tr = tid % TR, tc = tid / TR;
    const int n0 = blockIdx.x * BN, m0 = blockIdx.y * BM;
    // the order of the sums has whole chunks: an odd number of stages ends with one of zeros
    const int rank = GROUPS == 2 ? gf_rank() : 0, kbase = rank * GF_GROUP;
    const int klen = GROUPS == 2 ? min(K - kbase, GF_GROUP) : K;
    const int stages = 2 * ((klen + GF_CHUNK - 1) / GF_CHUNK);
    ng_pdl_trigger();

    auto load_w = [&](int t) {
        float* s = gt_smem + (t % GT_STAGES) * STAGE + BM * GT_ROW;
#pragma unroll
        for (int i = tid; i < BN * (GT_BK / 4); i += 128) {
            const int r = i / (GT_BK / 4), k = (i % (GT_BK / 4)) * 4, kk = kbase + t * GT_BK + k;
            const int have = n0 + r < N ? K - kk : 0;
            gf_copy4<AL>(s + r * GT_ROW + k, have > 0 ? W + (size_t)(n0 + r) * ldw + kk : W, have);
        }
    };
    auto load_a = [&](int t, const float* a) {
        float* s = gt_smem + (t % GT_STAGES) * STAGE;
#pragma unroll
        for (int i = tid; i < BM * (GT_BK / 4); i += 128) {
            const int r = i / (GT_BK / 4), k = (i % (GT_BK / 4)) * 4, kk = kbase + t * GT_BK + k;
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
    float total[TM][TN], before[GROUPS == 1 ? TM : 1][GROUPS == 1 ? TN : 1];     // of the group, of the groups before it
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            acc[i][j] = 0ull, total[i][j] = 0.f;
            if constexpr (GROUPS == 1) before[i][j] = 0.f;
        }

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
            if constexpr (GROUPS == 1)
                if ((t + 1) % (GF_GROUP / GT_BK) == 0 || t + 1 == stages)        // a group's end
#pragma unroll
                    for (int i = 0; i < TM; ++i)
#pragma unroll
                        for (int j = 0; j < TN; ++j) before[i][j] += total[i][j], total[i][j] = 0.f;
        }
    }
    if constexpr (GROUPS == 1)
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN; ++j) total[i][j] = before[i][j];
    if constexpr (GROUPS == 2) {                                 // the blocks of a cluster: each adds up some rows of the tile
        static_assert(BM * BN <= GT_STAGES * STAGE, "the tile's sums fit where the stages were");
        __syncthreads();                                         // every stage has been read
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN; ++j) gt_smem[(tr + i * TR) * BN + tc + j * TC] = total[i][j];
        gf_cluster_sync();
        const int blocks = gridDim.z;
        for (int e = tid; e < ((BM - rank + blocks - 1) / blocks) * BN; e += 128) {
            const int r = rank + e / BN * blocks, c = e % BN, m = m0 + r, n = n0 + c;
            if (m >= M || n >= N) continue;
            float v[GF_MAX_CLUSTER], sum = 0.f;
#pragma unroll
            for (int b = 0; b < GF_MAX_CLUSTER; ++b) v[b] = b < blocks ? gf_peer(gt_smem + r * BN + c, b) : 0.f;
#pragma unroll
            for (int b = 0; b < GF_MAX_CLUSTER; ++b)
                if (b < blocks) sum += v[b];
            C[(size_t)m * ldc + n] = sum + (bias ? bias[n] : 0.f);
        }
        gf_cluster_sync();
        return;
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

// as ng_launch, the blocks of one (x, y) as a cluster
template <typename... KP, typename... A>
static int gf_launch_cluster(void (*kernel)(KP...), dim3 grid, int threads, size_t smem, cudaStream_t stream, A... args) {
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    memset(attr, 0, sizeof(attr));
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = grid.z;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = ng_pdl_enabled() ? 2 : 1;
    cudaLaunchKernelEx(&cfg, kernel, KP(args)...);
    return ng_launch_status();
}

template <int MR, bool AL, bool CLUSTER>
static int gf_rows_as(const float* A, const float* W, const float* bias, float* C, int M, int N, int K, int lda, int ldw,
                      int ldc, cudaStream_t stream) {
    const int groups = gf_groups(K), stages = CLUSTER ? 1 : groups < GR_STAGES ? groups : GR_STAGES;
    constexpr int STAGE = GR_COLS * GR_WROW + MR * GR_XROW, PART = 2 * GR_CH * MR * GR_COLS;
    static std::atomic<unsigned long long> done{0};
    if (!ng_allow_smem(done, gemm_f32_rows_kernel<MR, AL, CLUSTER>, (GR_STAGES * STAGE + PART) * 4)) return NG_LAUNCH_FAILED;
    dim3 grid((N + GR_COLS - 1) / GR_COLS, (M + MR - 1) / MR, CLUSTER ? groups : 1);
    if (grid.y > 65535) return NG_BAD_SIZE;
    const size_t smem = (size_t)(stages * STAGE + PART) * 4;
    if (CLUSTER) return gf_launch_cluster(gemm_f32_rows_kernel<MR, AL, CLUSTER>, grid, GR_COLS * GR_CH, smem, stream, A, W, bias, C, M, N, K, lda, ldw, ldc, stages);
    NG_LAUNCH((gemm_f32_rows_kernel<MR, AL, CLUSTER>), grid, GR_COLS * GR_CH, smem, stream, A, W, bias, C, M, N, K, lda, ldw, ldc, stages);
    return ng_launch_status();
}
template <int MR, bool AL>
static int gf_rows(const float* A, const float* W, const float* bias, float* C, int M, int N, int K, int lda, int ldw,
                   int ldc, cudaStream_t stream) {
    if (gf_rows_cluster(M, N, K))
        return gf_rows_as<MR, AL, true>(A, W, bias, C, M, N, K, lda, ldw, ldc, stream);
    return gf_rows_as<MR, AL, false>(A, W, bias, C, M, N, K, lda, ldw, ldc, stream);
}

template <int BM, int BN, int TM, int TN, bool AL, int GROUPS>
static int gf_tile_as(const float* A, const float* W, const float* bias, float* C, int M, int N, int K, int lda, int ldw,
                      int ldc, cudaStream_t stream) {
    constexpr int BYTES = GT_STAGES * (BM + BN) * GT_ROW * 4;
    static std::atomic<unsigned long long> done{0};
    if (!ng_allow_smem(done, gemm_f32_tile_kernel<BM, BN, TM, TN, AL, GROUPS>, BYTES)) return NG_LAUNCH_FAILED;
    dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM, GROUPS == 2 ? gf_groups(K) : 1);
    if (grid.y > 65535) return NG_BAD_SIZE;
    if (GROUPS == 2) return gf_launch_cluster(gemm_f32_tile_kernel<BM, BN, TM, TN, AL, GROUPS>, grid, 128, BYTES, stream, A, W, bias, C, M, N, K, lda, ldw, ldc);
    NG_LAUNCH((gemm_f32_tile_kernel<BM, BN, TM, TN, AL, GROUPS>), grid, 128, BYTES, stream, A, W, bias, C, M, N, K, lda, ldw, ldc);
    return ng_launch_status();
}
template <int BM, int BN, int TM, int TN, bool AL>
static int gf_tile(const float* A, const float* W, const float* bias, float* C, int M, int N, int K, int lda, int ldw,
                   int ldc, cudaStream_t s) {
    if (gf_groups(K) == 1) return gf_tile_as<BM, BN, TM, TN, AL, 0>(A, W, bias, C, M, N, K, lda, ldw, ldc, s);
    if (gf_tile_cluster(M, N, K)) return gf_tile_as<BM, BN, TM, TN, AL, 2>(A, W, bias, C, M, N, K, lda, ldw, ldc, s);
    return gf_tile_as<BM, BN, TM, TN, AL, 1>(A, W, bias, C, M, N, K, lda, ldw, ldc, s);
}

// Rows up to which the few-rows kernel takes the product: it reads the weights once per 8 rows (from the L2 after the
// first time) with 128 blocks at N = 1,024, where 32-row tiles would leave 32 blocks to walk K alone.
#define GF_ROWS_MAX 32

template <bool AL>
static int gf_dispatch(const float* A, const float* W, const float* bias, float* C, int M, int N, int K, int lda,
                       int ldw, int ldc, cudaStream_t s) {
    if (M <= GF_ROWS_MAX) {
        switch (gf_rows_of_block(M)) {
            case 1: return gf_rows<1, AL>(A, W, bias, C, M, N, K, lda, ldw, ldc, s);
            case 2: return gf_rows<2, AL>(A, W, bias, C, M, N, K, lda, ldw, ldc, s);
            case 4: return gf_rows<4, AL>(A, W, bias, C, M, N, K, lda, ldw, ldc, s);
            default: return gf_rows<8, AL>(A, W, bias, C, M, N, K, lda, ldw, ldc, s);
        }
    }
    switch (gf_tile_size(M, N, K)) {
        case 0: return gf_tile<64, 64, 8, 4, AL>(A, W, bias, C, M, N, K, lda, ldw, ldc, s);
        case 1: return gf_tile<32, 64, 4, 4, AL>(A, W, bias, C, M, N, K, lda, ldw, ldc, s);
        default: return gf_tile<32, 32, 4, 2, AL>(A, W, bias, C, M, N, K, lda, ldw, ldc, s);
    }
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
