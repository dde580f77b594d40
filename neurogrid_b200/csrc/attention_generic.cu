// Paged attention for any query length, head size and dtype: the plain, order-fixed kernel.
//
// A block owns one (query row, head).  The visible keys lo..pos are cut into tiles of 8 at multiples of 8 positions;
// tile t belongs to warp t mod 4, which walks its tiles in ascending order with an online softmax, and the four
// warps' results are merged in order.  All of it depends on the row's position alone, so the result for a token does
// not depend on how the request was cut into steps or on what else is in the batch.  It is the whole float32 path
// and the in-GPU check for the tensor-core kernels of the bfloat16 path.
//
// Bound by the latency of the chain load - dot - softmax - sum, not by bytes or FMAs; hence eight keys at a time (their
// loads in flight together, one exponential a lane for all eight) and four chains a row: 23 us a launch where one warp
// walking the keys one by one took 185 us (350M LFM2 shape, 2 rows or 256 padded rows, about 100 keys, 16 heads of 64).
//
// Reference: gpu/cuda/paged_attention.cu:278-387 (decode, one block per head, all scores in
// shared memory, context <= 4096) and gpu/cuda/attention.cu:369-500 (prefill, materialised
// [heads, S, S] scores, K/V expanded to all query heads).  Both use scale 1/sqrt(hd), mask
// key > query, query head h reads KV head h / (nH / nKV).  `slopes` (one float per query head, or
// null) adds a position term to the scores: -slope[h] * (query position - key position).
#include "ng_common.cuh"

#define AG_WARPS 4
#define AG_TILE 8
#define AG_MAX_J 24     // head_dim <= 768

// MJ: columns a lane holds (head_dim <= 32 * MJ).  Z: more heads than a grid's second dimension has blocks, the third counts on (a form
// of its own: one more comparison in all of them cost heads of 257 and more a quarter of their speed)
template <typename T, int MJ, bool Z>
__global__ void __launch_bounds__(AG_WARPS * 32)
attention_generic_kernel(const T* __restrict__ q, const T* __restrict__ k_pages, const T* __restrict__ v_pages,
                         const int* __restrict__ table, int table_stride, const int* __restrict__ positions,
                         const int* __restrict__ row_entry, T* __restrict__ out, int nH, int nKV, int hd,
                         int page_size, int num_pages, int window, float scale, const float* __restrict__ slopes) {
    __shared__ float acc_s[AG_WARPS][32 * MJ], ml_s[2][AG_WARPS];
    ng_pdl_trigger();
    ng_pdl_wait();
    const int row = blockIdx.x, head = Z ? blockIdx.z * gridDim.y + blockIdx.y : blockIdx.y;
    if (Z && head >= nH) return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    T* o = out + ((size_t)row * nH + head) * hd;
    const int entry = row_entry[row];
    if (entry < 0) {
        for (int j = threadIdx.x; j < hd; j += AG_WARPS * 32) ng_st(o + j, 0.f);
        return;
    }
    const int pos = positions[row];
    const int kvh = head / (nH / nKV);
    const int lo = window > 0 ? max(0, pos - window + 1) : 0;
    const float slope = slopes ? slopes[head] : 0.f;          // score bias: -slope * (query position - key position)
    const T* qr = q + ((size_t)row * nH + head) * hd;
    float qv[MJ], acc[MJ];
#pragma unroll
    for (int j = 0; j < MJ; ++j) {
        const int d = lane + 32 * j;
        qv[j] = d < hd ? ng_ld(qr + d) * scale : 0.f;
        acc[j] = 0.f;
    }
    float m = -INFINITY, l = 0.f;
    const int* trow = table + (size_t)entry * table_stride;
    int t = lo / AG_TILE;
    t += (warp - t % AG_WARPS + AG_WARPS) % AG_WARPS;
    for (; t * AG_TILE <= pos; t += AG_WARPS) {
        // lane 4 i + (0..3) looks after key i of the tile
        const int kp = t * AG_TILE + (lane >> 2);
        long long base = -1;
        if (kp >= lo && kp <= pos) {
            const int page = trow[kp / page_size];
            if (page >= 0 && page < num_pages) base = (((long long)page * nKV + kvh) * page_size + kp % page_size) * hd;
        }
        float dot[AG_TILE];
#pragma unroll
        for (int i = 0; i < AG_TILE; ++i) {
            const long long b = __shfl_sync(0xffffffffu, base, 4 * i);
            dot[i] = 0.f;
#pragma unroll
            for (int j = 0; j < MJ; ++j) {
                const int d = lane + 32 * j;
                dot[i] = fmaf(qv[j], b >= 0 && d < hd ? ng_ld(k_pages + b + d) : 0.f, dot[i]);
            }
        }
        // eight sums over 32 lanes: each halving step keeps the half of the keys that the lane's bit names
#pragma unroll
        for (int o2 = 16, n = AG_TILE / 2; o2 >= 4; o2 >>= 1, n >>= 1)
#pragma unroll
            for (int i = 0; i < AG_TILE / 2; ++i)
                if (i < n) {
                    const bool up = lane & o2;
                    const float send = up ? dot[i] : dot[i + n], keep = up ? dot[i + n] : dot[i];
                    dot[i] = keep + __shfl_xor_sync(0xffffffffu, send, o2);
                }
        dot[0] += __shfl_xor_sync(0xffffffffu, dot[0], 2);
        dot[0] += __shfl_xor_sync(0xffffffffu, dot[0], 1);
        const float s = base >= 0 ? dot[0] - slope * (float)(pos - kp) : -INFINITY;
        float mt = s;
#pragma unroll
        for (int o2 = 4; o2 <= 16; o2 <<= 1) mt = fmaxf(mt, __shfl_xor_sync(0xffffffffu, mt, o2));
        const float m_new = fmaxf(m, mt);
        if (m_new == -INFINITY && !__any_sync(0xffffffffu, s != s)) continue;      // no key of the tile can be read
        const float corr = expf(m - m_new);
        const float p = base >= 0 ? expf(s - m_new) : 0.f;
        float pt = p;
#pragma unroll
        for (int o2 = 4; o2 <= 16; o2 <<= 1) pt += __shfl_xor_sync(0xffffffffu, pt, o2);
        l = l * corr + pt;
#pragma unroll
        for (int j = 0; j < MJ; ++j) acc[j] *= corr;
#pragma unroll
        for (int i = 0; i < AG_TILE; ++i) {
            const long long b = __shfl_sync(0xffffffffu, base, 4 * i);
            const float pi = __shfl_sync(0xffffffffu, p, 4 * i);
#pragma unroll
            for (int j = 0; j < MJ; ++j) {
                const int d = lane + 32 * j;
                acc[j] = fmaf(pi, b >= 0 && d < hd ? ng_ld(v_pages + b + d) : 0.f, acc[j]);
            }
        }
        m = m_new;
    }
#pragma unroll
    for (int j = 0; j < MJ; ++j) acc_s[warp][lane + 32 * j] = acc[j];
    if (lane == 0) ml_s[0][warp] = m, ml_s[1][warp] = l;
    __syncthreads();
    float top = ml_s[0][0], sum = 0.f, f[AG_WARPS];
#pragma unroll
    for (int w = 1; w < AG_WARPS; ++w) top = fmaxf(top, ml_s[0][w]);
#pragma unroll
    for (int w = 0; w < AG_WARPS; ++w) {
        // a warp without keys has m = -inf and sums of zero; one that met a NaN has it in its sums
        f[w] = ml_s[0][w] == -INFINITY ? 1.f : expf(ml_s[0][w] - top);
        sum += ml_s[1][w] * f[w];
    }
    const float inv = sum > 0.f ? 1.f / sum : 0.f;
    for (int d = threadIdx.x; d < hd; d += AG_WARPS * 32) {
        float v = 0.f;
#pragma unroll
        for (int w = 0; w < AG_WARPS; ++w) v += acc_s[w][d] * f[w];
        ng_st(o + d, v * inv);
    }
}

NG_EXPORT int ng_attention_generic(const void* q, const void* k_pages, const void* v_pages, const int* table,
                                   int table_stride, const int* positions, const int* row_entry, void* out,
                                   int n_rows, int nH, int nKV, int hd, int page_size, int num_pages, int window,
                                   float scale, const float* slopes, int act_bf16, cudaStream_t stream) {
    if (n_rows <= 0) return NG_OK;
    if (hd <= 0 || hd > 32 * AG_MAX_J || nH <= 0 || nKV <= 0 || nH % nKV || page_size <= 0) return NG_BAD_SIZE;
    dim3 grid(n_rows, nH < 65535 ? nH : 65535, (nH + 65534) / 65535);
    if (grid.z > 65535) return NG_BAD_SIZE;
#define AG_LAUNCH(TT, MJ, Z)                                                                                           \
    NG_LAUNCH((attention_generic_kernel<TT, MJ, Z>), grid, AG_WARPS * 32, 0, stream, (const TT*)q, (const TT*)k_pages, \
              (const TT*)v_pages, table, table_stride, positions, row_entry, (TT*)out, nH, nKV, hd, page_size, num_pages, \
              window, scale, slopes)
#define AG_SIZES(TT)                                                                                                   \
    do {                                                                                                               \
        if (grid.z > 1) AG_LAUNCH(TT, 24, true);                                                                       \
        else if (hd <= 64) AG_LAUNCH(TT, 2, false);                                                                    \
        else if (hd <= 128) AG_LAUNCH(TT, 4, false);                                                                   \
        else if (hd <= 256) AG_LAUNCH(TT, 8, false);                                                                   \
        else AG_LAUNCH(TT, 24, false);                                                                                 \
    } while (0)
    if (act_bf16) AG_SIZES(__nv_bfloat16);
    else AG_SIZES(float);
    return ng_launch_status();
}
