// Per-layer token input: x += rmsnorm(W_proj (gelu_tanh(W_gate x) * e[token])) * w.
//
//   x: the float32 residual stream [n_rows, H], complete (every pending sum added);
//   e: [vocab, dim] float32, the layer's columns of the token table;
//   W_gate [dim, H], W_proj^T [dim, H] (transposed when bound, so that both are read along H), w [H] float32.
// Everything is float32 FFMA.  Kernels for dim <= 64, H <= 2,048, H % 4 == 0 (few rows: a cluster; many: tiles) and for any
// size; in each a row's arithmetic does not depend on the other rows.
#include "ng_common.cuh"

__device__ __forceinline__ float gelu_tanh(float z) {
    return 0.5f * z * (1.f + tanhf(0.7978845608028654f * (z + 0.044715f * z * z * z)));
}
__device__ __forceinline__ uint64_t ts_fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ float ts_lo(uint64_t v) { return __uint_as_float((uint32_t)v); }
__device__ __forceinline__ float ts_hi(uint64_t v) { return __uint_as_float((uint32_t)(v >> 32)); }

// The row's token, and whether the row belongs to a request; a token outside the table is reported and read as 0.
__device__ __forceinline__ bool ts_row(const int* tokens, const int* row_entry, int row, int n_rows, int vocab, bool report,
                                       int* status, int& tok) {
    tok = 0;
    if (row >= n_rows || row_entry[row] < 0) return false;
    tok = tokens[row];
    if (tok < 0 || tok >= vocab) {
        if (report) atomicOr(status, NG_STATUS_BAD_TOKEN);
        tok = 0;
    }
    return true;
}

// ---- few rows --------------------------------------------------------------------------------------------------
// Bound by latency: three dependent sums over 1 MB of weights for a handful of rows.  A cluster of eight blocks takes
// R rows: each block forms an eighth of the gate values (a warp each) and hands them to the others through
// distributed shared memory, then an eighth of the columns of y and of the sum of squares, which is exchanged the same
// way.  One launch in place of three: 7.1 us inside a step's graph against 23 us (8 rows, H = 2048, dim = 64).  FIT (a warp's row of W_gate and a thread's column of W_proj fit its
// registers: dim <= 64, H <= 2048, H % 4 == 0): both (with four rows the former) are requested before the kernel in
// front has ended.
#define TC_BLOCKS 8
#define TC_THREADS 256
#define TC_WARPS (TC_THREADS / 32)
#define TC_NG 16                         // float4 a lane holds of a row of W_gate
#define TC_DIM 64

__device__ __forceinline__ uint32_t tc_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void tc_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void tc_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
// a float into the same place of another block's shared memory
__device__ __forceinline__ void tc_put(float* p, uint32_t block, float v) {
    uint32_t a = (uint32_t)__cvta_generic_to_shared(p), r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(block));
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(r), "f"(v) : "memory");
}

template <int R, bool FIT>
__global__ void __cluster_dims__(TC_BLOCKS, 1, 1) __launch_bounds__(TC_THREADS)
token_side_cluster_kernel(float* __restrict__ h_, const int* __restrict__ tokens, const float* __restrict__ table,
                          const float* __restrict__ w_gate, const float* __restrict__ w_proj_t,
                          const float* __restrict__ w_norm, int n_rows, int H, int dim, int vocab, float eps,
                          const int* __restrict__ row_entry, int* __restrict__ status, int cols) {
    extern __shared__ float ts_sm[];
    float* gs = ts_sm;                             // [R][dim]
    float* ys = ts_sm + R * dim;                   // [R][cols], where a thread has several columns (!FIT)
    __shared__ float ssp[R][TC_BLOCKS], red[TC_WARPS][R];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int rank = tc_rank(), r0 = (blockIdx.x / TC_BLOCKS) * R;
    const int per = (dim + TC_BLOCKS - 1) / TC_BLOCKS, i0 = rank * per, i1 = min(dim, i0 + per);
    const int c0 = rank * cols, c1 = min(H, c0 + cols);
    ng_pdl_trigger();
    float4 wg[FIT ? TC_NG : 1];
    constexpr bool PROJ = FIT && R == 1;           // four rows' sums leave no registers for the column as well
    float wp[PROJ ? TC_DIM : 1];
    if constexpr (FIT) {
        const bool mine = i0 + warp < i1;
#pragma unroll
        for (int k = 0; k < TC_NG; ++k) {
            const int j = lane * 4 + 128 * k;
            wg[k] = mine && j < H ? *reinterpret_cast<const float4*>(w_gate + (size_t)(i0 + warp) * H + j) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        if constexpr (PROJ)
#pragma unroll
            for (int i = 0; i < TC_DIM; ++i) wp[i] = i < dim && c0 + tid < c1 ? w_proj_t[(size_t)i * H + c0 + tid] : 0.f;
    }
    tc_arrive();                                   // the others' shared memory may be written once all have started
    ng_pdl_wait();
    float* h = ng_after_wait(h_);
    bool live[R];
    int tok[R];
#pragma unroll
    for (int r = 0; r < R; ++r) live[r] = ts_row(tokens, row_entry, r0 + r, n_rows, vocab, rank == 0 && tid == 0, status, tok[r]);
    tc_wait();
    for (int i = i0 + warp; i < i1; i += TC_WARPS) {
        float acc[R];
#pragma unroll
        for (int r = 0; r < R; ++r) acc[r] = 0.f;
        if constexpr (FIT) {
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const float* x = h + (size_t)min(r0 + r, n_rows - 1) * H;
#pragma unroll
                for (int k = 0; k < TC_NG; ++k) {
                    const int j = lane * 4 + 128 * k;
                    const float4 xv = j < H ? *reinterpret_cast<const float4*>(x + j) : make_float4(0.f, 0.f, 0.f, 0.f);
                    acc[r] = fmaf(xv.x, wg[k].x, fmaf(xv.y, wg[k].y, fmaf(xv.z, wg[k].z, fmaf(xv.w, wg[k].w, acc[r]))));
                }
            }
        } else {
            for (int j = lane; j < H; j += 32) {
                const float wv = w_gate[(size_t)i * H + j];
#pragma unroll
                for (int r = 0; r < R; ++r) acc[r] = fmaf(h[(size_t)min(r0 + r, n_rows - 1) * H + j], wv, acc[r]);
            }
        }
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const float a = ng_warp_sum(acc[r]);
            if (lane < TC_BLOCKS) tc_put(gs + r * dim + i, lane, gelu_tanh(a) * table[(size_t)tok[r] * dim + i]);
        }
    }
    tc_arrive();
    tc_wait();
    float ss[R], y[R];
#pragma unroll
    for (int r = 0; r < R; ++r) ss[r] = y[r] = 0.f;
    if constexpr (FIT) {
        if constexpr (PROJ) {
#pragma unroll
            for (int i = 0; i < TC_DIM; ++i)
                if (i < dim) y[0] = fmaf(wp[i], gs[i], y[0]);
        } else if (c0 + tid < c1) {
#pragma unroll 16
            for (int i = 0; i < dim; ++i) {
                const float wv = w_proj_t[(size_t)i * H + c0 + tid];
#pragma unroll
                for (int r = 0; r < R; ++r) y[r] = fmaf(wv, gs[r * dim + i], y[r]);
            }
        }
#pragma unroll
        for (int r = 0; r < R; ++r) ss[r] = y[r] * y[r];
    } else {
        for (int c = c0 + tid; c < c1; c += TC_THREADS) {
            float acc[R];
#pragma unroll
            for (int r = 0; r < R; ++r) acc[r] = 0.f;
#pragma unroll 8
            for (int i = 0; i < dim; ++i) {
                const float wv = w_proj_t[(size_t)i * H + c];
#pragma unroll
                for (int r = 0; r < R; ++r) acc[r] = fmaf(wv, gs[r * dim + i], acc[r]);
            }
#pragma unroll
            for (int r = 0; r < R; ++r) {
                ys[r * cols + c - c0] = acc[r];
                ss[r] += acc[r] * acc[r];
            }
        }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const float s = ng_warp_sum(ss[r]);
        if (lane == 0) red[warp][r] = s;
    }
    __syncthreads();
    if (tid < TC_BLOCKS * R) {
        const int r = tid / TC_BLOCKS;
        float s = 0.f;
#pragma unroll
        for (int k = 0; k < TC_WARPS; ++k) s += red[k][r];
        tc_put(&ssp[r][rank], tid % TC_BLOCKS, s);
    }
    tc_arrive();
    tc_wait();
#pragma unroll
    for (int r = 0; r < R; ++r) {
        if (!live[r]) continue;
        float s = 0.f;
#pragma unroll
        for (int k = 0; k < TC_BLOCKS; ++k) s += ssp[r][k];
        const float f = rsqrtf(s / (float)H + eps);
        for (int c = c0 + tid; c < c1; c += TC_THREADS)
            h[(size_t)(r0 + r) * H + c] += (FIT ? y[r] : ys[r * cols + c - c0]) * f * w_norm[c];
    }
}

// ---- many rows -------------------------------------------------------------------------------------------------
// Bound by the FMA pipe (2 * 2 * dim * H operations a row) once the matrices come through shared memory: read from the L2
// straight into registers, rows H apart, they cost 20 wavefronts a load and the kernel 60 us (2,048 rows of 1,024), now 36 us;
// 93 us for one that read shared memory for every FMA.  A block takes 16 rows, staged in shared memory; both matrices pass through one
// ring of 17 KB stages, TL_STAGES - 1 ahead.  Gate: a stage is 64 k of W_gate; each of the eight warps takes eight of them and
// forms all 16 x 64 values over its k, 4 x 8 a lane (even and odd k in the halves of a packed FMA); the warps' sums are
// added in order.  Projection: a stage is four rows of 1,024 columns of W_proj^T; a thread owns four neighbouring columns (NC
// times) for all 16 rows and keeps y in registers until the row's mean square is known.
#define TL_ROWS 16
#define TL_THREADS 256
#define TL_WARPS (TL_THREADS / 32)
#define TL_DIM 64
#define TL_COLS (4 * TL_THREADS)
#define TL_STAGES 4
#define TL_KS 64                         // k of a gate stage
#define TL_PITCH (TL_KS + 4)             // eight rows' 16 bytes in different banks
#define TL_STAGE (TL_DIM * TL_PITCH)
#define TL_PI 4                          // rows of W_proj^T of a stage
static_assert(TL_PI * TL_COLS <= TL_STAGE, "a stage holds either");

__host__ __device__ constexpr int tl_rows_floats(int H) {          // the rows; the warps' sums take their place
    return TL_ROWS * (H + 4) > TL_WARPS * TL_ROWS * TL_DIM ? TL_ROWS * (H + 4) : TL_WARPS * TL_ROWS * TL_DIM;
}
// 16 bytes to shared memory, asynchronously; zeros where `real` is false
__device__ __forceinline__ void tl_copy(float* dst, const float* src, bool real) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(real ? 16 : 0) : "memory");
}

template <int NC>
__global__ void __launch_bounds__(TL_THREADS, 1)
token_side_tile_kernel(float* __restrict__ h_, const int* __restrict__ tokens, const float* __restrict__ table,
                       const float* __restrict__ w_gate, const float* __restrict__ w_proj_t,
                       const float* __restrict__ w_norm, int n_rows, int H, int dim, int vocab, float eps,
                       const int* __restrict__ row_entry, int* __restrict__ status) {
    extern __shared__ __align__(16) float ts_sm[];
    const int ldx = H + 4;                                         // rows 4 words apart modulo the banks
    float* xs = ts_sm;                                             // [16][H + 4]
    float* part = ts_sm;                                           // then [8 warps][16][64]
    float* ring = ts_sm + tl_rows_floats(H);                       // [TL_STAGES][TL_STAGE]
    float2* g2 = reinterpret_cast<float2*>(ring + TL_STAGES * TL_STAGE);            // [64][16]: (g, g)
    __shared__ int s_tok[TL_ROWS], s_live[TL_ROWS];
    __shared__ float red[TL_WARPS][TL_ROWS], scale[TL_ROWS];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int r0 = blockIdx.x * TL_ROWS, rg = lane >> 3, cg = lane & 7;
    const int gate_stages = (H + TL_KS - 1) / TL_KS, pieces = (dim + TL_PI - 1) / TL_PI, stages = gate_stages + NC * pieces;
    ng_pdl_trigger();
    auto request = [&](int t) {                                    // one group of copies a stage, empty ones at the end
        float* s = ring + (t % TL_STAGES) * TL_STAGE;
        if (t < gate_stages) {
#pragma unroll
            for (int q = 0; q < TL_DIM * TL_KS / 4 / TL_THREADS; ++q) {
                const int i = tid + q * TL_THREADS, r = i / (TL_KS / 4), k = (i % (TL_KS / 4)) * 4;
                const bool real = r < dim && t * TL_KS + k < H;
                tl_copy(s + r * TL_PITCH + k, real ? w_gate + (size_t)r * H + t * TL_KS + k : w_gate, real);
            }
        } else if (t < stages) {
            const int c = (t - gate_stages) / pieces, i0 = ((t - gate_stages) % pieces) * TL_PI, col = c * TL_COLS + tid * 4;
#pragma unroll
            for (int q = 0; q < TL_PI; ++q) {
                const bool real = i0 + q < dim && col < H;
                tl_copy(s + q * TL_COLS + tid * 4, real ? w_proj_t + (size_t)(i0 + q) * H + col : w_proj_t, real);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    // stage t has landed and the one read before it may be written again
    auto next = [&](int t) {
        asm volatile("cp.async.wait_group %0;" ::"n"(TL_STAGES - 2) : "memory");
        __syncthreads();
        request(t + TL_STAGES - 1);
        return ring + (t % TL_STAGES) * TL_STAGE;
    };
    for (int t = 0; t < TL_STAGES - 1; ++t) request(t);
    ng_pdl_wait();
    float* h = ng_after_wait(h_);
    if (tid < TL_ROWS) {
        int tok;
        s_live[tid] = ts_row(tokens, row_entry, r0 + tid, n_rows, vocab, true, status, tok);
        s_tok[tid] = tok;
    }
    __syncthreads();
#pragma unroll 8
    for (int i = tid; i < TL_ROWS * (H / 4); i += TL_THREADS) {
        const int r = i / (H / 4), j = (i % (H / 4)) * 4;
        *reinterpret_cast<float4*>(xs + r * ldx + j) =
            s_live[r] ? *reinterpret_cast<const float4*>(h + (size_t)(r0 + r) * H + j) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    {
        uint64_t acc[4][8];
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int j = 0; j < 8; ++j) acc[r][j] = 0ull;
        for (int t = 0; t < gate_stages; ++t) {
            const float* w = next(t) + cg * TL_PITCH + warp * 8;
            const int k = t * TL_KS + warp * 8;
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                if (k + 4 * q >= H) break;                         // (the rows end there)
                ulonglong2 xv[4];
#pragma unroll
                for (int r = 0; r < 4; ++r) xv[r] = *reinterpret_cast<const ulonglong2*>(xs + (4 * r + rg) * ldx + k + 4 * q);
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const ulonglong2 wv = *reinterpret_cast<const ulonglong2*>(w + 8 * j * TL_PITCH + 4 * q);
#pragma unroll
                    for (int r = 0; r < 4; ++r) acc[r][j] = ts_fma2(xv[r].y, wv.y, ts_fma2(xv[r].x, wv.x, acc[r][j]));
                }
            }
        }
        __syncthreads();                                           // the rows are done with
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int j = 0; j < 8; ++j)
                part[(warp * TL_ROWS + 4 * r + rg) * TL_DIM + cg + 8 * j] = ts_lo(acc[r][j]) + ts_hi(acc[r][j]);
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < TL_ROWS * TL_DIM / TL_THREADS; ++q) {
        const int i = tid + q * TL_THREADS, r = i / TL_DIM, d = i % TL_DIM;
        float a = 0.f;
#pragma unroll
        for (int k = 0; k < TL_WARPS; ++k) a += part[(k * TL_ROWS + r) * TL_DIM + d];
        const float g = d < dim ? gelu_tanh(a) * table[(size_t)s_tok[r] * dim + d] : 0.f;
        g2[d * TL_ROWS + r] = make_float2(g, g);
    }
    __syncthreads();
    uint64_t y[NC][TL_ROWS][2];
#pragma unroll
    for (int c = 0; c < NC; ++c) {
#pragma unroll
        for (int r = 0; r < TL_ROWS; ++r) y[c][r][0] = y[c][r][1] = 0ull;
        for (int t = 0; t < pieces; ++t) {
            const float* w = next(gate_stages + c * pieces + t) + tid * 4;
#pragma unroll
            for (int q = 0; q < TL_PI; ++q) {                      // (rows beyond dim are zeros, and so are their g)
                const ulonglong2 wv = *reinterpret_cast<const ulonglong2*>(w + q * TL_COLS);
                const ulonglong2* gp = reinterpret_cast<const ulonglong2*>(g2 + (t * TL_PI + q) * TL_ROWS);
#pragma unroll
                for (int r = 0; r < TL_ROWS; r += 2) {
                    const ulonglong2 gv = gp[r / 2];
                    y[c][r][0] = ts_fma2(gv.x, wv.x, y[c][r][0]);
                    y[c][r][1] = ts_fma2(gv.x, wv.y, y[c][r][1]);
                    y[c][r + 1][0] = ts_fma2(gv.y, wv.x, y[c][r + 1][0]);
                    y[c][r + 1][1] = ts_fma2(gv.y, wv.y, y[c][r + 1][1]);
                }
            }
        }
    }
#pragma unroll
    for (int r = 0; r < TL_ROWS; ++r) {
        float s = 0.f;
#pragma unroll
        for (int c = 0; c < NC; ++c)
#pragma unroll
            for (int p = 0; p < 2; ++p) s += ts_lo(y[c][r][p]) * ts_lo(y[c][r][p]) + ts_hi(y[c][r][p]) * ts_hi(y[c][r][p]);
        s = ng_warp_sum(s);
        if (lane == 0) red[warp][r] = s;
    }
    __syncthreads();
    if (tid < TL_ROWS) {
        float s = 0.f;
#pragma unroll
        for (int k = 0; k < TL_WARPS; ++k) s += red[k][tid];
        scale[tid] = rsqrtf(s / (float)H + eps);
    }
    __syncthreads();
#pragma unroll
    for (int c = 0; c < NC; ++c) {
        const int col = c * TL_COLS + tid * 4;
        if (col >= H) continue;
        const float4 w = *reinterpret_cast<const float4*>(w_norm + col);
#pragma unroll
        for (int r = 0; r < TL_ROWS; ++r) {
            if (!s_live[r]) continue;
            float4* hp = reinterpret_cast<float4*>(h + (size_t)(r0 + r) * H + col);
            const float4 x = *hp;
            const float f = scale[r];
            *hp = make_float4(x.x + ts_lo(y[c][r][0]) * f * w.x, x.y + ts_hi(y[c][r][0]) * f * w.y,
                              x.z + ts_lo(y[c][r][1]) * f * w.z, x.w + ts_hi(y[c][r][1]) * f * w.w);
        }
    }
}

// ---- any size --------------------------------------------------------------------------------------------------
// A block takes R rows (8 or 4 for long steps, so that the two matrices are read once per so many rows; 1 for short ones): the
// rows are staged in shared memory, a warp per gate value forms the R dot products, then a thread per column forms y for the
// R rows, which replaces the staged rows; the mean squares are reduced per row and the sum goes into the stream.  Bound by
// shared memory (read for every FMA).  `aligned`: rows of H % 4 == 0 take 16-byte accesses.
template <int R, int TS_THREADS>
__global__ void __launch_bounds__(TS_THREADS)
token_side_kernel(float* __restrict__ h, const int* __restrict__ tokens, const float* __restrict__ table,
                  const float* __restrict__ w_gate, const float* __restrict__ w_proj_t, const float* __restrict__ w_norm,
                  int n_rows, int H, int dim, int vocab, float eps, const int* __restrict__ row_entry,
                  int* __restrict__ status, int aligned) {
    extern __shared__ float sm[];
    float* buf = sm;                 // [R][H]: the rows, then y
    float* g = sm + (size_t)R * H;   // [R][dim]
    __shared__ float red[R][TS_THREADS / 32];
    __shared__ float scale[R];
    ng_pdl_trigger();
    ng_pdl_wait();
    const int r0 = blockIdx.x * R;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int NW = TS_THREADS / 32;
    bool live[R];
    int tok[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        live[r] = r0 + r < n_rows && row_entry[r0 + r] >= 0;
        tok[r] = live[r] ? tokens[r0 + r] : 0;
        if (tok[r] < 0 || tok[r] >= vocab) {
            if (tid == 0) atomicOr(status, NG_STATUS_BAD_TOKEN);
            tok[r] = 0;
        }
    }
#pragma unroll
    for (int r = 0; r < R; ++r)
        for (int j = tid; j < H; j += TS_THREADS) buf[(size_t)r * H + j] = live[r] ? h[(size_t)(r0 + r) * H + j] : 0.f;
    __syncthreads();
    const bool vec = aligned && (H % 4) == 0;            // rows of the matrices start on 16-byte boundaries
    for (int i = warp; i < dim; i += NW) {
        const float* w = w_gate + (size_t)i * H;
        float acc[R];
#pragma unroll
        for (int r = 0; r < R; ++r) acc[r] = 0.f;
        if (vec) {
#pragma unroll 4
            for (int j = lane * 4; j < H; j += 128) {
                const float4 wv = *reinterpret_cast<const float4*>(w + j);
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const float4 xv = *reinterpret_cast<const float4*>(buf + (size_t)r * H + j);
                    acc[r] = fmaf(xv.x, wv.x, fmaf(xv.y, wv.y, fmaf(xv.z, wv.z, fmaf(xv.w, wv.w, acc[r]))));
                }
            }
        } else {
            for (int j = lane; j < H; j += 32) {
                const float wv = w[j];
#pragma unroll
                for (int r = 0; r < R; ++r) acc[r] = fmaf(buf[(size_t)r * H + j], wv, acc[r]);
            }
        }
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const float a = ng_warp_sum(acc[r]);
            if (lane == 0) g[r * dim + i] = gelu_tanh(a) * table[(size_t)tok[r] * dim + i];
        }
    }
    __syncthreads();
    float ss[R];
#pragma unroll
    for (int r = 0; r < R; ++r) ss[r] = 0.f;
    if (vec) {
        for (int j = tid * 4; j < H; j += 4 * TS_THREADS) {          // four columns a thread
            float4 acc[R];
#pragma unroll
            for (int r = 0; r < R; ++r) acc[r] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
            for (int i = 0; i < dim; ++i) {
                const float4 wv = *reinterpret_cast<const float4*>(w_proj_t + (size_t)i * H + j);
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const float gv = g[r * dim + i];
                    acc[r].x = fmaf(wv.x, gv, acc[r].x);
                    acc[r].y = fmaf(wv.y, gv, acc[r].y);
                    acc[r].z = fmaf(wv.z, gv, acc[r].z);
                    acc[r].w = fmaf(wv.w, gv, acc[r].w);
                }
            }
#pragma unroll
            for (int r = 0; r < R; ++r) {
                *reinterpret_cast<float4*>(buf + (size_t)r * H + j) = acc[r];
                ss[r] += acc[r].x * acc[r].x + acc[r].y * acc[r].y + acc[r].z * acc[r].z + acc[r].w * acc[r].w;
            }
        }
    } else {
        for (int j = tid; j < H; j += TS_THREADS) {
            float acc[R];
#pragma unroll
            for (int r = 0; r < R; ++r) acc[r] = 0.f;
            for (int i = 0; i < dim; ++i) {
                const float wv = w_proj_t[(size_t)i * H + j];
#pragma unroll
                for (int r = 0; r < R; ++r) acc[r] = fmaf(wv, g[r * dim + i], acc[r]);
            }
#pragma unroll
            for (int r = 0; r < R; ++r) {
                buf[(size_t)r * H + j] = acc[r];
                ss[r] += acc[r] * acc[r];
            }
        }
    }
    __syncthreads();                                     // the sum below reads columns other threads wrote
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const float s = ng_warp_sum(ss[r]);
        if (lane == 0) red[r][warp] = s;
    }
    __syncthreads();
    if (tid < R) {
        float s = 0.f;
        for (int k = 0; k < NW; ++k) s += red[tid][k];
        scale[tid] = rsqrtf(s / (float)H + eps);
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < R; ++r) {
        if (!live[r]) continue;
        float* hr = h + (size_t)(r0 + r) * H;
        for (int j = tid; j < H; j += TS_THREADS) hr[j] += buf[(size_t)r * H + j] * scale[r] * w_norm[j];
    }
}

// Few rows: a block per row would leave most of the GPU idle and stream both matrices through one SM, so the same sums
// are dealt to many blocks: `gate` forms eight gate values a block (a warp each, the same walk as above), `proj` forms y for 128
// columns a block and the partial sum of their squares, `apply` adds up the partial sums in ascending order and adds the
// normed y into the stream.  `scratch`: g [n_rows, dim], y [n_rows, H], partial sums [n_rows, ceil(H / 128)], float32.
__global__ void __launch_bounds__(256)
token_side_gate_kernel(const float* __restrict__ h, const int* __restrict__ tokens, const float* __restrict__ table,
                       const float* __restrict__ w_gate, float* __restrict__ g, int H, int dim, int vocab,
                       const int* __restrict__ row_entry, int* __restrict__ status, int aligned) {
    ng_pdl_trigger();
    ng_pdl_wait();
    const int row = blockIdx.y, lane = threadIdx.x & 31;
    const int i = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (i >= dim || row_entry[row] < 0) return;
    int tok = tokens[row];
    if (tok < 0 || tok >= vocab) {
        if (lane == 0) atomicOr(status, NG_STATUS_BAD_TOKEN);
        tok = 0;
    }
    const float* x = h + (size_t)row * H;
    const float* w = w_gate + (size_t)i * H;
    float acc = 0.f;
    if (aligned && H % 4 == 0) {
#pragma unroll 4
        for (int j = lane * 4; j < H; j += 128) {
            const float4 wv = *reinterpret_cast<const float4*>(w + j), xv = *reinterpret_cast<const float4*>(x + j);
            acc = fmaf(xv.x, wv.x, fmaf(xv.y, wv.y, fmaf(xv.z, wv.z, fmaf(xv.w, wv.w, acc))));
        }
    } else {
        for (int j = lane; j < H; j += 32) acc = fmaf(x[j], w[j], acc);
    }
    acc = ng_warp_sum(acc);
    if (lane == 0) g[(size_t)row * dim + i] = gelu_tanh(acc) * table[(size_t)tok * dim + i];
}

__global__ void __launch_bounds__(128)
token_side_proj_kernel(const float* __restrict__ g, const float* __restrict__ w_proj_t, float* __restrict__ y,
                       float* __restrict__ ss_part, int H, int dim, int n_slices, const int* __restrict__ row_entry) {
    __shared__ float red[32];
    ng_pdl_trigger();
    ng_pdl_wait();
    const int row = blockIdx.y;
    if (row_entry[row] < 0) return;
    const int j = blockIdx.x * 128 + threadIdx.x;
    const float* gr = g + (size_t)row * dim;
    float acc = 0.f;
    if (j < H) {
#pragma unroll 8
        for (int i = 0; i < dim; ++i) acc = fmaf(w_proj_t[(size_t)i * H + j], gr[i], acc);
        y[(size_t)row * H + j] = acc;
    }
    const float ss = ng_block_sum(acc * acc, red);
    if (threadIdx.x == 0) ss_part[(size_t)row * n_slices + blockIdx.x] = ss;
}

__global__ void __launch_bounds__(256)
token_side_apply_kernel(float* __restrict__ h, const float* __restrict__ y, const float* __restrict__ ss_part,
                        const float* __restrict__ w_norm, int H, int n_slices, float eps, const int* __restrict__ row_entry) {
    ng_pdl_trigger();
    ng_pdl_wait();
    const int row = blockIdx.x;
    if (row_entry[row] < 0) return;
    float ss = 0.f;
    for (int k = 0; k < n_slices; ++k) ss += ss_part[(size_t)row * n_slices + k];
    const float r = rsqrtf(ss / (float)H + eps);
    for (int j = threadIdx.x; j < H; j += blockDim.x) h[(size_t)row * H + j] += y[(size_t)row * H + j] * r * w_norm[j];
}

template <int R, int TS_THREADS>
static int token_side_launch(float* h, const int* tokens, const float* table, const float* w_gate, const float* w_proj_t,
                             const float* w_norm, const int* row_entry, int n_rows, int H, int dim, int vocab, float eps,
                             int* status, int vec, cudaStream_t stream) {
    const size_t smem = (size_t)R * ((size_t)H + dim) * sizeof(float);
    static bool configured = false;
    if (!configured) {
        if (cudaFuncSetAttribute(token_side_kernel<R, TS_THREADS>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024) != cudaSuccess)
            return NG_LAUNCH_FAILED;
        configured = true;
    }
    NG_LAUNCH((token_side_kernel<R, TS_THREADS>), (n_rows + R - 1) / R, TS_THREADS, smem, stream, h, tokens, table, w_gate, w_proj_t,
              w_norm, n_rows, H, dim, vocab, eps, row_entry, status, vec);
    return ng_launch_status();
}

// ---- which ------------------------------------------------------------------------------------------------------
// us for 8 / 64 / 255 / 400 / 1,024 / 2,048 rows:
//   H = 1,024, dim = 64:  cluster (FIT) 5.5 / 10.2 / 21.9 / - / - / -, blocks of rows - / - / 23.5 / 26.2 / 37.8 / 73.5, tiles - / - / 35.0 / 36.5 / 36.1 / 36.1
//   H = 2,048, dim = 64:  cluster (FIT) 6.1 / 14.3 / 29.1 / - / - / -, blocks of rows - / - / 29.9 / 38.6 / 47.9 / 93.6, tiles - / - / 68.0 / 69.9 / 70.1 / 70.4
//   H = 1,024, dim = 256: cluster 48 / 38 / 51 / 85 / 182 / 359, three kernels 28 / 33 / -, blocks of rows - / - / 74 / 88 / 115 / 226
//   H = 2,049, dim = 64:  cluster 24 / 32 / 37 / 66 / 135 / 256, three kernels 20 / 20 / -, blocks of rows - / - / 45 / 59 / 65 / 128
//   H = 4,096, dim = 64:  cluster 35 / 56 / 63 / 111 / 211 / 390, three kernels 20 / 26 / -, blocks of rows - / - / 46 / 66 / 76 / 149
// Sizes that a cluster's registers hold: a cluster for up to TS_FEW rows; tiles are worth their 16 rows a block once blocks of
// eight rows need a second round of the SMs, and from 512 rows on where a thread has four columns only (H <= 1,024).
#define TS_FEW 255
#define TS_SCRATCH_ROWS 128              // fewer rows than this of any size: the three kernels, if the caller has scratch
#define TS_ROW_CAP (160 * 1024)          // bytes of rows that a block stages

static bool ts_fits(int H, int dim) { return dim <= TL_DIM && H <= 2 * TL_COLS && H % 4 == 0; }

NG_EXPORT int ng_token_side(float* h, const int* tokens, const float* table, const float* w_gate, const float* w_proj_t,
                            const float* w_norm, const int* row_entry, int n_rows, int H, int dim, int vocab, float eps,
                            int* status, float* scratch, cudaStream_t stream) {
    if (n_rows <= 0) return NG_OK;
    if (H <= 0 || dim <= 0 || vocab <= 0) return NG_BAD_SIZE;
    const bool wide = H % 4 == 0 && (((uintptr_t)h | (uintptr_t)w_gate | (uintptr_t)w_proj_t | (uintptr_t)w_norm) & 15) == 0;
    const int cols = ((H + TC_BLOCKS - 1) / TC_BLOCKS + 3) & ~3;
#define TC_GO(R, FIT)                                                                                                  \
    do {                                                                                                               \
        const size_t smem = (size_t)R * (dim + (FIT ? 0 : cols)) * sizeof(float);                                      \
        NG_LAUNCH((token_side_cluster_kernel<R, FIT>), ((n_rows + R - 1) / R) * TC_BLOCKS, TC_THREADS, smem, stream, h, tokens, \
                  table, w_gate, w_proj_t, w_norm, n_rows, H, dim, vocab, eps, row_entry, status, cols);               \
        return ng_launch_status();                                                                                     \
    } while (0)
    // 16 rows are 128 blocks; beyond them a cluster's blocks read the weights once per four rows
    if (wide && ts_fits(H, dim) && n_rows <= TS_FEW) {
        if (n_rows <= 16) TC_GO(1, true);
        TC_GO(4, true);
    }
    // other sizes, where blocks of four rows would have few columns or single-element accesses each
    if (n_rows >= TS_SCRATCH_ROWS && n_rows < (H <= TL_COLS ? 600 : 400) && (H <= TL_COLS || !wide) && !(wide && ts_fits(H, dim)) &&
        4 * ((size_t)dim + cols) * sizeof(float) <= 48 * 1024)
        TC_GO(4, false);
    if (wide && ts_fits(H, dim) && (n_rows > 8 * 148 || (H <= TL_COLS && n_rows >= 512))) {
        const size_t smem = (size_t)(tl_rows_floats(H) + TL_STAGES * TL_STAGE + 2 * TL_DIM * TL_ROWS) * sizeof(float);
        const int blocks = (n_rows + TL_ROWS - 1) / TL_ROWS;
#define TL_GO(NC)                                                                                                      \
    do {                                                                                                               \
        static bool configured = false;                                                                                \
        if (!configured) {                                                                                             \
            if (cudaFuncSetAttribute(token_side_tile_kernel<NC>, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024) != cudaSuccess) \
                return NG_LAUNCH_FAILED;                                                                               \
            configured = true;                                                                                         \
        }                                                                                                              \
        NG_LAUNCH((token_side_tile_kernel<NC>), blocks, TL_THREADS, smem, stream, h, tokens, table, w_gate, w_proj_t, w_norm, \
                  n_rows, H, dim, vocab, eps, row_entry, status);                                                      \
        return ng_launch_status();                                                                                     \
    } while (0)
        if (H <= TL_COLS) TL_GO(1);
        TL_GO(2);
    }
    const size_t per_row = ((size_t)H + dim) * sizeof(float);
    if (scratch && (n_rows < TS_SCRATCH_ROWS || per_row > TS_ROW_CAP)) {
        const int n_slices = (H + 127) / 128;
        if (n_rows > 65535) return NG_BAD_SIZE;
        float* g = scratch;
        float* y = g + (size_t)n_rows * dim;
        float* part = y + (size_t)n_rows * H;
        NG_LAUNCH((token_side_gate_kernel), dim3((dim + 7) / 8, n_rows), 256, 0, stream, (const float*)h, tokens, table, w_gate,
                  g, H, dim, vocab, row_entry, status, (int)wide);
        NG_LAUNCH((token_side_proj_kernel), dim3(n_slices, n_rows), 128, 0, stream, (const float*)g, w_proj_t, y, part, H, dim,
                  n_slices, row_entry);
        NG_LAUNCH((token_side_apply_kernel), n_rows, 256, 0, stream, h, (const float*)y, (const float*)part, w_norm, H,
                  n_slices, eps, row_entry);
        return ng_launch_status();
    }
    if (per_row > TS_ROW_CAP) return NG_BAD_SIZE;
#define TS_GO(RR, TT) return token_side_launch<RR, TT>(h, tokens, table, w_gate, w_proj_t, w_norm, row_entry, n_rows, H, dim, vocab, eps, status, (int)wide, stream)
    if (n_rows >= 512 && 8 * per_row <= TS_ROW_CAP) TS_GO(8, 512);
    if (n_rows >= 128 && 4 * per_row <= TS_ROW_CAP) TS_GO(4, 512);
    TS_GO(1, 1024);            // few rows: a block's speed is its loads in flight
}
