// Input convolution of a sublayer: out[t] = u[t] + sum_{k<L} w[d,k] * u[t-(L-1)+k] per channel d,
// over a ragged batch of prompt portions and single tokens (tap L-1 multiplies the current token).
// u before the first row of a portion comes from the request's state slot (its last L-1 inputs,
// float32), u before position 0 is zero whatever the slot holds; after the portion the slot holds
// the last L-1 inputs again.
//
// Grid: (channel blocks, token tiles, entries).  A thread owns one channel of one tile and walks
// its tokens in order with the last L-1 inputs in registers.  Only tile 0 of an entry reads the
// slot and only tile 0 writes it, after all its reads: no other block touches a slot in use.
// The sum is float32, taps ascending, so a token's result does not depend on the cut.
#include "ng_common.cuh"

#define IC_MAX_L 8
#define IC_TILE 32
#define IC_THREADS 128

template <typename T, int L>
__global__ void __launch_bounds__(IC_THREADS)
input_conv_kernel(const T* __restrict__ u, const float* __restrict__ w, float* __restrict__ state,
                  T* __restrict__ out, const int* __restrict__ cu_q, const int* __restrict__ ctx_before,
                  const int* __restrict__ slots, int H) {
    ng_pdl_trigger();
    ng_pdl_wait();
    const int e = blockIdx.z;
    const int q0 = cu_q[e];
    const int qlen = cu_q[e + 1] - q0;
    const int t0 = blockIdx.y * IC_TILE;
    const int d = blockIdx.x * IC_THREADS + threadIdx.x;
    if (t0 >= qlen || d >= H) return;
    const int ctx = ctx_before[e];
    float* st = state + (size_t)slots[e] * (L - 1) * H + d;        // st[j*H]: u at position ctx-(L-1)+j
    const T* ur = u + (size_t)q0 * H + d;
    T* orow = out + (size_t)q0 * H + d;
    float wk[L], hist[L - 1], old[L - 1];
#pragma unroll
    for (int k = 0; k < L; ++k) wk[k] = w[(size_t)d * L + k];
    const bool first = t0 == 0;
#pragma unroll
    for (int j = 0; j < L - 1; ++j)
        old[j] = (first && ctx - (L - 1) + j >= 0) ? st[(size_t)j * H] : 0.f;
    // hist[j] = u at chunk index t0-(L-1)+j
#pragma unroll
    for (int j = 0; j < L - 1; ++j) {
        const int ti = t0 - (L - 1) + j;
        hist[j] = ti >= 0 ? ng_ld(ur + (size_t)ti * H) : old[j];
    }
    const int t1 = min(t0 + IC_TILE, qlen);
    for (int t = t0; t < t1; ++t) {
        const float x = ng_ld(ur + (size_t)t * H);
        float acc = 0.f;
#pragma unroll
        for (int k = 0; k < L - 1; ++k)
            acc = fmaf(wk[k], hist[k], acc);
        acc = fmaf(wk[L - 1], x, acc);
        ng_st(orow + (size_t)t * H, x + acc);
#pragma unroll
        for (int k = 0; k < L - 2; ++k)
            hist[k] = hist[k + 1];
        hist[L - 2] = x;
    }
    if (first) {
        // the slot after the portion: u at positions ctx+qlen-(L-1)+j, from the portion or from what the slot held
#pragma unroll
        for (int j = 0; j < L - 1; ++j) {
            const int ti = qlen - (L - 1) + j;
            float v = 0.f;
            if (ti >= 0) v = ng_ld(ur + (size_t)ti * H);
            else {
#pragma unroll
                for (int k = 0; k < L - 1; ++k)
                    if (k == ti + (L - 1)) v = old[k];
            }
            st[(size_t)j * H] = v;
        }
    }
}

// The norm of the stream and the convolution behind it for single tokens (no entry has more than one): a block per row, a
// thread NV x 4 channels, the residual sum in front as in add_rmsnorm, whose arithmetic and order this is, and the
// convolution's of the kernel above.  A step of few rows is a chain of launches that wait for one another: two of them in
// one, everything but the stream (weights, taps, the slot) read before the wait.  A row of no entry gets its norm.
// The next launch may begin only after the wait: with a product that began earlier, beside it, the token input in front (a
// cluster, token_side.cu) took 12.3 us instead of 7.6, more than the product's head start gave.  Decode steps of 16
// layers behind 40 tokens, two launches / one that lets the next begin at its top / this one, us: width 2,048, 1 row 1,097 /
// 1,199 / 1,046, 4 rows 1,134 / 1,206 / 1,064, 8 rows 1,160 / 1,094 / 1,087, 64 rows 1,868 / 1,774 / 1,753; width 1,024, 1 row 843 /
// 765 / 693, 8 rows 854 / 802 / 722, 64 rows 1,231 / 1,159 / 1,131.
__device__ __forceinline__ float4 ic_ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 ic_ld4(const __nv_bfloat16* p) {
    const uint2 u = *reinterpret_cast<const uint2*>(p);
    const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.x)), b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.y));
    return make_float4(a.x, a.y, b.x, b.y);
}
__device__ __forceinline__ void ic_st4(float* p, const float (&v)[4]) { *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]); }
__device__ __forceinline__ void ic_st4(__nv_bfloat16* p, const float (&v)[4]) {
    const __nv_bfloat162 a = __floats2bfloat162_rn(v[0], v[1]), b = __floats2bfloat162_rn(v[2], v[3]);
    uint2 u;
    u.x = *reinterpret_cast<const uint32_t*>(&a);
    u.y = *reinterpret_cast<const uint32_t*>(&b);
    *reinterpret_cast<uint2*>(p) = u;
}
template <typename T> __device__ __forceinline__ float ic_round(float v) {
    T r;
    ng_st(&r, v);
    return ng_ld(&r);
}

template <typename TD, typename T, int L, int NV>
__global__ void __launch_bounds__(256)
norm_conv_token_kernel(float* __restrict__ h, const TD* __restrict__ delta, const float* __restrict__ nw, const float* __restrict__ w,
                       float* __restrict__ state, T* __restrict__ out, const int* __restrict__ row_entry,
                       const int* __restrict__ ctx_before, const int* __restrict__ slots, int H, float eps, int n_partials,
                       size_t partial_stride) {
    __shared__ float red[32];
    const int row = blockIdx.x, entry = row_entry[row];                  // the batch description: older than the step's kernels
    const int ctx = entry >= 0 ? ctx_before[entry] : 0;
    float* st = state + (size_t)(entry >= 0 ? slots[entry] : 0) * (L - 1) * H;
    float* hr = h + (size_t)row * H;
    float4 v[NV], ww[NV], old[NV][L - 1];
    float taps[NV][4 * L];
#pragma unroll
    for (int u = 0; u < NV; ++u) {
        const int j = 4 * (threadIdx.x + u * blockDim.x);
        const bool in = j < H;
        ww[u] = in ? ic_ld4(nw + j) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int k = 0; k < L; ++k) {
            const float4 t = in ? ic_ld4(w + (size_t)j * L + 4 * k) : make_float4(0.f, 0.f, 0.f, 0.f);
            taps[u][4 * k] = t.x; taps[u][4 * k + 1] = t.y; taps[u][4 * k + 2] = t.z; taps[u][4 * k + 3] = t.w;
        }
#pragma unroll
        for (int k = 0; k < L - 1; ++k)
            old[u][k] = in && entry >= 0 && ctx - (L - 1) + k >= 0 ? ic_ld4(st + (size_t)k * H + j) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    ng_pdl_wait();
    ng_pdl_trigger();                                                    // not earlier: see above
    delta = ng_after_wait(delta);
    float ss = 0.f;
#pragma unroll
    for (int u = 0; u < NV; ++u) {
        const int j = 4 * (threadIdx.x + u * blockDim.x);
        v[u] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (j < H) {
            v[u] = ic_ld4(hr + j);
            if (delta) {
                for (int s = 0; s < n_partials; ++s) {                   // ascending s: a fixed order
                    const float4 d = ic_ld4(delta + s * partial_stride + (size_t)row * H + j);
                    v[u].x += d.x; v[u].y += d.y; v[u].z += d.z; v[u].w += d.w;
                }
                *reinterpret_cast<float4*>(hr + j) = v[u];
            }
            ss += v[u].x * v[u].x + v[u].y * v[u].y + v[u].z * v[u].z + v[u].w * v[u].w;
        }
    }
    ss = ng_block_sum(ss, red);
    const float r = rsqrtf(ss / (float)H + eps);
#pragma unroll
    for (int u = 0; u < NV; ++u) {
        const int j = 4 * (threadIdx.x + u * blockDim.x);
        if (j >= H) continue;
        const float x[4] = {ic_round<T>(v[u].x * r * ww[u].x), ic_round<T>(v[u].y * r * ww[u].y), ic_round<T>(v[u].z * r * ww[u].z),
                            ic_round<T>(v[u].w * r * ww[u].w)};
        float y[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float acc = 0.f;
#pragma unroll
            for (int k = 0; k < L - 1; ++k) {
                const float4 o = old[u][k];
                acc = fmaf(taps[u][i * L + k], i == 0 ? o.x : i == 1 ? o.y : i == 2 ? o.z : o.w, acc);
            }
            acc = fmaf(taps[u][i * L + L - 1], x[i], acc);
            y[i] = entry >= 0 ? x[i] + acc : x[i];
        }
        ic_st4(out + (size_t)row * H + j, y);
        if (entry >= 0) {
#pragma unroll
            for (int k = 0; k < L - 2; ++k) *reinterpret_cast<float4*>(st + (size_t)k * H + j) = old[u][k + 1];
            *reinterpret_cast<float4*>(st + (size_t)(L - 2) * H + j) = make_float4(x[0], x[1], x[2], x[3]);
        }
    }
}

// h[row] (+= delta[row]: one [n, H] tensor of the activation type, or n_partials float32 ones partial_stride apart), then
// out[row] = u + conv(u) for u = rmsnorm(h[row]) nw; the slots take u.  For steps without an entry of more than one row.
// H a multiple of 4 up to 2,048 (a thread holds two pieces at most), every operand 16-byte aligned.
NG_EXPORT int ng_norm_input_conv(float* h, const void* delta, const float* nw, const float* w, float* state, void* out,
                                 const int* row_entry, const int* ctx_before, const int* slots, int n_rows, int H, int L, float eps,
                                 int act_bf16, int delta_f32, int n_partials, long long partial_stride, cudaStream_t stream) {
    if (n_rows <= 0) return NG_OK;
    if (H <= 0 || H % 4 || H > 2048 || L < 2 || L > 4 || n_partials < 1 || (n_partials > 1 && (!delta_f32 || partial_stride % 4)) ||
        (((uintptr_t)h | (uintptr_t)delta | (uintptr_t)nw | (uintptr_t)w | (uintptr_t)state | (uintptr_t)out) & 15))
        return NG_BAD_SIZE;
    const int threads = H <= 512 ? 128 : 256, nv = (H / 4 + threads - 1) / threads;
    const size_t ps = (size_t)partial_stride;
#define NC_GO(TD, T, LL, NV) NG_LAUNCH((norm_conv_token_kernel<TD, T, LL, NV>), n_rows, threads, 0, stream, h, (const TD*)delta, nw, w, \
                                       state, (T*)out, row_entry, ctx_before, slots, H, eps, n_partials, ps)
#define NC_TYPES(LL, NV)                                                             \
    do {                                                                             \
        if (act_bf16 && delta_f32) NC_GO(float, __nv_bfloat16, LL, NV);              \
        else if (act_bf16) NC_GO(__nv_bfloat16, __nv_bfloat16, LL, NV);              \
        else NC_GO(float, float, LL, NV);                                            \
    } while (0)
#define NC_CASE(LL) case LL: if (nv <= 1) NC_TYPES(LL, 1); else NC_TYPES(LL, 2); break;
    switch (L) { NC_CASE(2) NC_CASE(3) NC_CASE(4) }
    return ng_launch_status();
}

// u, out: [n_rows, H] of the activation type; w: [H, L] float32; state: [slots, L-1, H] float32.
NG_EXPORT int ng_input_conv(const void* u, const float* w, float* state, void* out, const int* cu_q,
                            const int* ctx_before, const int* slots, int n_entries, int max_q, int H, int L,
                            int act_bf16, cudaStream_t stream) {
    if (n_entries <= 0 || max_q <= 0) return NG_OK;
    if (H <= 0 || L < 2 || L > IC_MAX_L) return NG_BAD_SIZE;
    dim3 grid((H + IC_THREADS - 1) / IC_THREADS, (max_q + IC_TILE - 1) / IC_TILE, n_entries);
    if (grid.y > 65535 || grid.z > 65535) return NG_BAD_SIZE;
#define IC_CASE(LL)                                                                                                   \
    case LL:                                                                                                          \
        if (act_bf16)                                                                                                 \
            NG_LAUNCH((input_conv_kernel<__nv_bfloat16, LL>), grid, IC_THREADS, 0, stream, (const __nv_bfloat16*)u, w, \
                      state, (__nv_bfloat16*)out, cu_q, ctx_before, slots, H);                                        \
        else                                                                                                          \
            NG_LAUNCH((input_conv_kernel<float, LL>), grid, IC_THREADS, 0, stream, (const float*)u, w, state,         \
                      (float*)out, cu_q, ctx_before, slots, H);                                                       \
        break;
    switch (L) {
        IC_CASE(2) IC_CASE(3) IC_CASE(4) IC_CASE(5) IC_CASE(6) IC_CASE(7) IC_CASE(8)
    }
    return ng_launch_status();
}
