// Routed experts: the router and the weighting of the experts' activations.
//
// moe_router: logits z = W_r x + b in float32 (x is the activation row, W_r and b float32); the top_k
//   experts with the largest logits are chosen (of equal logits the lower index) and weighted by the
//   softmax over the chosen logits.  Output: dense weights [n_rows, n_experts] float32, zero for the
//   experts a row does not use.
// moe_scale: act[row, e*ff + j] *= weights[row, e] for the first n_experts*ff columns of an activation
//   row of width ld (what lies behind them, a shared expert's columns, stays as it is).  With the
//   weights applied, one product with all experts' down projections side by side is the weighted sum.
#include "ng_common.cuh"

#define MOE_MAX_TOP 32

__device__ __forceinline__ float4 moe_ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 moe_ld4(const __nv_bfloat16* p) {
    const uint2 u = *reinterpret_cast<const uint2*>(p);
    const __nv_bfloat162 a = *reinterpret_cast<const __nv_bfloat162*>(&u.x), b = *reinterpret_cast<const __nv_bfloat162*>(&u.y);
    return make_float4(__low2float(a), __high2float(a), __low2float(b), __high2float(b));
}

// The choice among a row's logits z[E], by one warp, an expert a lane: top_k times the largest logit not chosen yet, of
// equal ones the lower index (and, as a plain walk from index 0 has it, the first one left if that is not a number);
// the chosen ones' softmax goes to out[E], zeros elsewhere.
__device__ __forceinline__ void moe_choose(const float* z, float* out, int E, int top_k) {
    const int lane = threadIdx.x & 31;
    for (int e = lane; e < E; e += 32) out[e] = 0.f;
    __syncwarp();
    int mine = -1;                             // lane k keeps the k-th choice
    float val = 0.f;
    for (int k = 0; k < top_k; ++k) {
        float bv = -INFINITY;
        int bi = 0x7fffffff, first = 0x7fffffff;
        for (int e0 = 0; e0 < E; e0 += 32) {
            const int e = e0 + lane;
            bool taken = e >= E;
            for (int m = 0; m < k; ++m) taken |= __shfl_sync(0xffffffffu, mine, m) == e;
            const float v = taken ? -INFINITY : z[e];
            if (!taken && (v > bv || (v == bv && e < bi))) { bv = v; bi = e; }
            if (!taken) first = min(first, e);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
            const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
            if (ov > bv || (ov == bv && oi < bi)) { bv = ov; bi = oi; }
        }
        first = __reduce_min_sync(0xffffffffu, first);
        if (z[first] != z[first]) { bi = first; bv = z[first]; }
        if (lane == k) { mine = bi; val = bv; }
    }
    const float top = __shfl_sync(0xffffffffu, val, 0);         // the largest
    val = expf(val - top);
    float sum = 0.f;
    for (int k = 0; k < top_k; ++k) sum += __shfl_sync(0xffffffffu, val, k);
    if (lane < top_k) out[mine] = val / sum;
}

// Few rows: bound by latency (a round trip to memory for the dot products, then the choices one after the other).  A
// block per row, a warp per expert; HELD: a lane holds 2,048 columns of the expert's weights in its registers, the first
// of them requested before the kernel in front has ended, and the choice is a warp's instead of a thread's walk over all
// experts: 5.1 us a launch of 8 rows of 2,048 and 16 experts inside a step's graph against 14.6 us.  So many registers leave an
// SM one block; where rows come in many rounds of the SMs, four warps a row that read the weights as they go are faster
// (2,048 rows, 64 experts of 1,024 / 4,096 columns: 53 / 146 us against 139 / 241).  In these kernels and the next a
// lane adds its columns in ascending order: the logits' bits depend on H alone.
#define MR_NI 16                            // float4 a lane holds of an expert's weights
template <typename T, bool HELD>
__global__ void __launch_bounds__(HELD ? 512 : 128)
moe_router_kernel(const T* __restrict__ x_, const float* __restrict__ wr, const float* __restrict__ br,
                  float* __restrict__ weights, int H, int E, int top_k) {
    extern __shared__ float z[];               // [E]
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
    const int row = blockIdx.x;
    const bool wide = H % 4 == 0;              // four columns a lane and load
    const float4 none = make_float4(0.f, 0.f, 0.f, 0.f);
    float4 w[HELD ? MR_NI : 1];
    auto load_w = [&](int e, int i0) {
#pragma unroll
        for (int k = 0; k < (HELD ? MR_NI : 0); ++k) {
            const int i = i0 + lane * 4 + 128 * k;
            w[k] = wide && e < E && i < H ? moe_ld4(wr + (size_t)e * H + i) : none;
        }
    };
    ng_pdl_trigger();
    load_w(warp, 0);
    ng_pdl_wait();
    const T* x = ng_after_wait(x_) + (size_t)row * H;
    for (int e = warp; e < E; e += nwarp) {
        float acc = 0.f;
        if (wide && !HELD) {
#pragma unroll 4
            for (int i = lane * 4; i < H; i += 128) {
                const float4 xv = moe_ld4(x + i), wv = moe_ld4(wr + (size_t)e * H + i);
                acc = fmaf(xv.x, wv.x, fmaf(xv.y, wv.y, fmaf(xv.z, wv.z, fmaf(xv.w, wv.w, acc))));
            }
        } else if (wide) {
            for (int i0 = 0; i0 < H; i0 += 128 * MR_NI) {
#pragma unroll
                for (int k = 0; k < MR_NI; ++k) {
                    const int i = i0 + lane * 4 + 128 * k;
                    const float4 xv = i < H ? moe_ld4(x + i) : none;
                    acc = fmaf(xv.x, w[k].x, fmaf(xv.y, w[k].y, fmaf(xv.z, w[k].z, fmaf(xv.w, w[k].w, acc))));
                }
                if (i0 + 128 * MR_NI < H) load_w(e, i0 + 128 * MR_NI);
                else if (e + nwarp < E) load_w(e + nwarp, 0);
            }
        } else {
            for (int i = lane; i < H; i += 32) acc = fmaf(ng_ld(x + i), wr[(size_t)e * H + i], acc);
        }
        acc = ng_warp_sum(acc);
        if (lane == 0) z[e] = acc + (br ? br[e] : 0.f);
    }
    __syncthreads();
    if (warp == 0) moe_choose(z, weights + (size_t)row * E, E, top_k);
}

// Many rows: a block keeps W_r in shared memory, a warp takes whole rows: sixteen experts' sums at a time, then the choice.
// 2,048 rows of 1,024, 16 experts: 10.7 us; four rows a block of the kernel above take 38 us, one row a block with W_r read
// from the L2 by every row's block 25 us.
#define MRR_WARPS 16
template <typename T>
__global__ void __launch_bounds__(MRR_WARPS * 32, 1)
moe_router_rows_kernel(const T* __restrict__ x_, const float* __restrict__ wr, const float* __restrict__ br,
                       float* __restrict__ weights, int n_rows, int H, int E, int top_k) {
    extern __shared__ __align__(16) float mr_smem[];
    float* ws = mr_smem;                       // [E][H]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    float* z = mr_smem + (size_t)E * H + (size_t)warp * E;
    ng_pdl_trigger();
    for (int i = tid; i < E * H / 4; i += MRR_WARPS * 32) {
        const uint32_t d = (uint32_t)__cvta_generic_to_shared(ws + 4 * (size_t)i);
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(wr + 4 * (size_t)i) : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    ng_pdl_wait();
    const T* x = ng_after_wait(x_);
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    for (int row = blockIdx.x * MRR_WARPS + warp; row < n_rows; row += gridDim.x * MRR_WARPS) {
        const T* xr = x + (size_t)row * H;
        for (int e0 = 0; e0 < E; e0 += 16) {
            float acc[16];
#pragma unroll
            for (int e = 0; e < 16; ++e) acc[e] = 0.f;
#pragma unroll 4
            for (int i = lane * 4; i < H; i += 128) {
                const float4 xv = moe_ld4(xr + i);
#pragma unroll
                for (int e = 0; e < 16; ++e) {
                    if (e0 + e < E) {
                        const float4 w = moe_ld4(ws + (size_t)(e0 + e) * H + i);
                        acc[e] = fmaf(xv.x, w.x, fmaf(xv.y, w.y, fmaf(xv.z, w.z, fmaf(xv.w, w.w, acc[e]))));
                    }
                }
            }
#pragma unroll
            for (int e = 0; e < 16; ++e)
                if (e0 + e < E) {
                    const float a = ng_warp_sum(acc[e]);
                    if (lane == 0) z[e0 + e] = a + (br ? br[e0 + e] : 0.f);
                }
        }
        __syncwarp();
        moe_choose(z, weights + (size_t)row * E, E, top_k);
        __syncwarp();
    }
}

template <typename T>
__global__ void moe_scale_kernel(T* __restrict__ act, const float* __restrict__ weights, int n_rows, int E, int ff, int ld,
                                 int ldw, int cols) {
    // columns behind E*ff (a shared expert's) are reached only when its gate, weights[row, E], multiplies them
    ng_pdl_trigger();
    ng_pdl_wait();
    const int row = blockIdx.y;
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= cols) return;
    T* p = act + (size_t)row * ld + c;
    ng_st(p, ng_ld(p) * weights[(size_t)row * ldw + (c < E * ff ? c / ff : E)]);
}

// out[row, c] = silu(gate_up[row, c]) * gate_up[row, I + c] * (c < E*ff ? weights[row, c / ff] : 1): the SwiGLU of all
// experts side by side with the routing weight applied at once (steps whose gate/up product has no fused epilogue).
// `shared_gated`: the columns behind E*ff (a shared expert's) are multiplied by weights[row, E].  Rows of `weights`
// lie ldw apart.
template <typename T>
__global__ void moe_swiglu_scaled_kernel(const T* __restrict__ gate_up, const float* __restrict__ weights,
                                         T* __restrict__ out, int I, int E, int ff, int ldw, int shared_gated) {
    ng_pdl_trigger();
    ng_pdl_wait();
    const int row = blockIdx.y;
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= I) return;
    const float g = ng_ld(gate_up + (size_t)row * 2 * I + c), u = ng_ld(gate_up + (size_t)row * 2 * I + I + c);
    T act;
    ng_st(&act, g / (1.f + expf(-g)) * u);           // rounded as the unweighted activation is, then weighted
    const float w = c < E * ff ? weights[(size_t)row * ldw + c / ff] : (shared_gated ? weights[(size_t)row * ldw + E] : 1.f);
    ng_st(out + (size_t)row * I + c, ng_ld(&act) * w);
}

// the same, eight columns a thread with 16-byte accesses (bfloat16; I and ff multiples of 8, so that the eight share an expert)
__global__ void moe_swiglu_scaled_vec_kernel(const __nv_bfloat16* __restrict__ gate_up, const float* __restrict__ weights,
                                             __nv_bfloat16* __restrict__ out, int I, int E, int ff, int ldw, int shared_gated) {
    ng_pdl_trigger();
    ng_pdl_wait();
    const int row = blockIdx.y;
    const int c = (blockIdx.x * blockDim.x + threadIdx.x) * 8;
    if (c >= I) return;
    const uint4 gv = *reinterpret_cast<const uint4*>(gate_up + (size_t)row * 2 * I + c);
    const uint4 uv = *reinterpret_cast<const uint4*>(gate_up + (size_t)row * 2 * I + I + c);
    const float w = c < E * ff ? weights[(size_t)row * ldw + c / ff] : (shared_gated ? weights[(size_t)row * ldw + E] : 1.f);
    const __nv_bfloat16* g = reinterpret_cast<const __nv_bfloat16*>(&gv);
    const __nv_bfloat16* u = reinterpret_cast<const __nv_bfloat16*>(&uv);
    uint4 ov;
    __nv_bfloat16* o = reinterpret_cast<__nv_bfloat16*>(&ov);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const float gk = __bfloat162float(g[k]);
        const __nv_bfloat16 act = __float2bfloat16_rn(gk / (1.f + expf(-gk)) * __bfloat162float(u[k]));
        o[k] = __float2bfloat16_rn(__bfloat162float(act) * w);
    }
    *reinterpret_cast<uint4*>(out + (size_t)row * I + c) = ov;
}

NG_EXPORT int ng_moe_swiglu_scaled(const void* gate_up, const float* weights, void* out, int n_rows, int I, int E, int ff,
                                   int ldw, int shared_gated, int act_bf16, cudaStream_t stream) {
    if (n_rows <= 0) return NG_OK;
    if (E <= 0 || ff <= 0 || I < E * ff || n_rows > 65535 || ldw < E + (shared_gated ? 1 : 0)) return NG_BAD_SIZE;
    if (act_bf16 && I % 8 == 0 && ff % 8 == 0 && ((uintptr_t)gate_up & 15) == 0 && ((uintptr_t)out & 15) == 0) {
        dim3 vgrid((I / 8 + 127) / 128, n_rows);
        NG_LAUNCH((moe_swiglu_scaled_vec_kernel), vgrid, 128, 0, stream, (const __nv_bfloat16*)gate_up, weights,
                  (__nv_bfloat16*)out, I, E, ff, ldw, shared_gated);
        return ng_launch_status();
    }
    dim3 grid((I + 255) / 256, n_rows);
    if (act_bf16)
        NG_LAUNCH((moe_swiglu_scaled_kernel<__nv_bfloat16>), grid, 256, 0, stream, (const __nv_bfloat16*)gate_up, weights,
                  (__nv_bfloat16*)out, I, E, ff, ldw, shared_gated);
    else
        NG_LAUNCH((moe_swiglu_scaled_kernel<float>), grid, 256, 0, stream, (const float*)gate_up, weights, (float*)out, I, E, ff,
                  ldw, shared_gated);
    return ng_launch_status();
}

NG_EXPORT int ng_moe_router(const void* x, const float* wr, const float* br, float* weights, int n_rows, int H,
                            int E, int top_k, int act_bf16, cudaStream_t stream) {
    if (n_rows <= 0) return NG_OK;
    if (H <= 0 || E <= 0 || top_k < 1 || top_k > E || top_k > MOE_MAX_TOP || E > 8192) return NG_BAD_SIZE;
    // from 256 rows on (512 of more than 2,048 columns: 256 rows, 8 experts of 4,096 16.3 us, a block a row 6.6), where W_r fits a
    // block's shared memory and its rows allow 16-byte copies
    const size_t held = ((size_t)E * H + (size_t)MRR_WARPS * E) * sizeof(float);
    if (n_rows >= (H > 2048 ? 512 : 256) && H % 4 == 0 && held <= 200 * 1024 && ((uintptr_t)wr & 15) == 0) {
        int blocks = (n_rows + MRR_WARPS - 1) / MRR_WARPS;
        if (blocks > 148) blocks = 148;
#define MRR_GO(T)                                                                                                      \
    do {                                                                                                               \
        static std::atomic<unsigned long long> done{0};                                                                \
        if (!ng_allow_smem(done, moe_router_rows_kernel<T>, 200 * 1024)) return NG_LAUNCH_FAILED;                      \
        NG_LAUNCH((moe_router_rows_kernel<T>), blocks, MRR_WARPS * 32, held, stream, (const T*)x, wr, br, weights, n_rows, H, E, top_k); \
        return ng_launch_status();                                                                                     \
    } while (0)
        if (act_bf16) MRR_GO(__nv_bfloat16);
        MRR_GO(float);
    }
    const int threads = 32 * (E < 4 ? 4 : E > 16 ? 16 : E);
    const size_t smem = (size_t)E * sizeof(float);
    // 1,024 rows: 64 experts of 1,024 columns 71 us with held weights, 51 without; of 4,096 121 and 130; 16 of 4,096 45 and 35
    const int held_rows = H <= 1024 || E <= 16 ? 512 : 1024;
#define MR_GO(T)                                                                                                       \
    do {                                                                                                               \
        if (n_rows <= held_rows)                                                                                       \
            NG_LAUNCH((moe_router_kernel<T, true>), n_rows, threads, smem, stream, (const T*)x, wr, br, weights, H, E, top_k); \
        else                                                                                                           \
            NG_LAUNCH((moe_router_kernel<T, false>), n_rows, 128, smem, stream, (const T*)x, wr, br, weights, H, E, top_k); \
    } while (0)
    if (act_bf16) MR_GO(__nv_bfloat16);
    else MR_GO(float);
    return ng_launch_status();
}

NG_EXPORT int ng_moe_scale(void* act, const float* weights, int n_rows, int E, int ff, int ld, int ldw, int shared_gated,
                           int act_bf16, cudaStream_t stream) {
    if (n_rows <= 0) return NG_OK;
    if (E <= 0 || ff <= 0 || ld < E * ff || n_rows > 65535 || ldw < E + (shared_gated ? 1 : 0)) return NG_BAD_SIZE;
    const int cols = shared_gated ? ld : E * ff;
    dim3 grid((cols + 255) / 256, n_rows);
    if (act_bf16)
        NG_LAUNCH((moe_scale_kernel<__nv_bfloat16>), grid, 256, 0, stream, (__nv_bfloat16*)act, weights, n_rows, E, ff, ld, ldw, cols);
    else
        NG_LAUNCH((moe_scale_kernel<float>), grid, 256, 0, stream, (float*)act, weights, n_rows, E, ff, ld, ldw, cols);
    return ng_launch_status();
}

// ------------------------------------------------------------------------------------------ sigmoid scores, groups
// moe_router_sigmoid: scores s = sigmoid(W_r x) in float32.  Choice scores are s + correction (no correction: s); the
//   experts form n_groups equal groups of neighbours, a group's score is the sum of its two largest choice scores (of
//   its one score where a group is one expert), and only experts of the keep_groups best groups can be chosen (of equal
//   scores the lower index wins, for groups and for experts).  The top_k chosen experts are weighted by their scores s
//   (without the correction) over their sum + 1e-20.  Output: dense weights [n_rows, ldw], zero for experts a row does
//   not use; with `wsg` (float32 [H]) column E receives sigmoid(wsg . x), the gate of a shared expert.
//   `softmax_scores`: s = softmax(W_r x) over all experts instead of the sigmoid.  `group_max`: a group's score is its
//   largest choice score.  `route_scale` multiplies the weights.
//   `n_identity`: the last that many of the E experts are the identity; they take part in scores, choice and sum like the
//   others but have no column of their own, the sum of their weights goes to one column behind the others (and behind the
//   shared expert's gate, if there is one).
template <typename T>
__global__ void __launch_bounds__(512)
moe_router_sigmoid_kernel(const T* __restrict__ x, const float* __restrict__ wr, const float* __restrict__ corr,
                          const float* __restrict__ wsg, float* __restrict__ weights, int H, int E, int ldw, int top_k,
                          int n_groups, int keep_groups, int softmax_scores, int group_max, float route_scale, int n_identity) {
    extern __shared__ float z[];               // [E] scores s, [E] choice scores, [n_groups] group scores
    float* choice = z + E;
    float* gscore = choice + E;
    ng_pdl_trigger();
    ng_pdl_wait();
    const int row = blockIdx.x;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
    const T* xr = x + (size_t)row * H;
    float* out = weights + (size_t)row * ldw;
    const int n_own = E - n_identity;          // experts with a column
    for (int e = warp; e < E + (wsg ? 1 : 0); e += nwarp) {
        const float* w = e < E ? wr + (size_t)e * H : wsg;
        float acc = 0.f;
        if (H % 4 == 0) {
#pragma unroll 4
            for (int i = lane * 4; i < H; i += 128) {
                const float4 xv = moe_ld4(xr + i), wv = moe_ld4(w + i);
                acc = fmaf(xv.x, wv.x, fmaf(xv.y, wv.y, fmaf(xv.z, wv.z, fmaf(xv.w, wv.w, acc))));
            }
        } else {
            for (int i = lane; i < H; i += 32) acc = fmaf(ng_ld(xr + i), w[i], acc);
        }
        acc = ng_warp_sum(acc);
        if (lane == 0) {
            const float s = 1.f / (1.f + expf(-acc));
            if (e < E) { z[e] = softmax_scores ? acc : s; choice[e] = s + (corr ? corr[e] : 0.f); if (e < n_own) out[e] = 0.f; }
            else out[n_own] = s;
        }
    }
    __syncthreads();
    if (softmax_scores) {                  // the first warp: largest logit, the exponentials' sum in index order per lane
        if (warp == 0) {
            float mx = -INFINITY;
            for (int e = lane; e < E; e += 32) mx = fmaxf(mx, z[e]);
            mx = ng_warp_max(mx);
            float sum = 0.f;
            for (int e = lane; e < E; e += 32) sum += expf(z[e] - mx);
            sum = ng_warp_sum(sum);
            for (int e = lane; e < E; e += 32) {
                const float s = expf(z[e] - mx) / sum;
                z[e] = s;
                choice[e] = s + (corr ? corr[e] : 0.f);
            }
        }
        __syncthreads();
    }
    const int per = E / n_groups;
    for (int g = threadIdx.x; g < n_groups; g += blockDim.x) {
        float a = -INFINITY, b = -INFINITY;             // the two largest of the group
        for (int e = g * per; e < (g + 1) * per; ++e) {
            const float v = choice[e];
            if (v > a) { b = a; a = v; } else if (v > b) b = v;
        }
        gscore[g] = per > 1 && !group_max ? a + b : a;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        if (keep_groups < n_groups) {
            // a group stays when fewer than keep_groups groups come before it (a larger score, or an equal one at a lower index)
            for (int g = 0; g < n_groups; ++g) {
                int ahead = 0;
                for (int o = 0; o < n_groups; ++o) ahead += (gscore[o] > gscore[g]) || (gscore[o] == gscore[g] && o < g);
                if (ahead >= keep_groups)
                    for (int e = g * per; e < (g + 1) * per; ++e) choice[e] = -INFINITY;
            }
        }
    }
    if (warp != 0) return;
    __syncwarp();
    // the first warp, one expert a round: every lane the best of its experts, then the best of the lanes; of equal choice
    // scores the lower index
    int mine = 0;                                // lane k: the k-th chosen expert
    float sum = 0.f;
    for (int k = 0; k < top_k; ++k) {
        float bv = -INFINITY;
        int best = E;
        for (int e = lane; e < E; e += 32) {
            const float v = choice[e];
            if (v > bv || (v == bv && e < best)) { bv = v; best = e; }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
            const int oe = __shfl_xor_sync(0xffffffffu, best, o);
            if (ov > bv || (ov == bv && oe < best)) { bv = ov; best = oe; }
        }
        best = min(best, E - 1);                 // (scores that are no numbers: some expert all the same)
        if (lane == k) mine = best;
        sum += z[best];
        __syncwarp();
        if (lane == 0) choice[best] = -INFINITY;
        __syncwarp();
    }
    const float w = lane < top_k ? z[mine] / (sum + 1e-20f) * route_scale : 0.f;
    const bool own = mine < n_own;
    if (lane < top_k && own) out[mine] = w;
    if (n_identity) {
        const float identity = ng_warp_sum(own ? 0.f : w);
        if (lane == 0) out[n_own + (wsg ? 1 : 0)] = identity;
    }
}

NG_EXPORT int ng_moe_router_sigmoid(const void* x, const float* wr, const float* corr, const float* wsg, float* weights,
                                    int n_rows, int H, int E, int ldw, int top_k, int n_groups, int keep_groups,
                                    int softmax_scores, int group_max, float route_scale, int n_identity, int act_bf16,
                                    cudaStream_t stream) {
    if (n_rows <= 0) return NG_OK;
    if (H <= 0 || E <= 0 || top_k < 1 || top_k > E || top_k > MOE_MAX_TOP || E > 4096 || n_groups < 1 || E % n_groups ||
        keep_groups < 1 || keep_groups > n_groups || top_k > keep_groups * (E / n_groups) || n_identity < 0 || n_identity > E ||
        ldw < E - n_identity + (wsg ? 1 : 0) + (n_identity ? 1 : 0))
        return NG_BAD_SIZE;
    const size_t smem = (size_t)(2 * E + n_groups) * sizeof(float);
    const int threads = n_rows <= 64 ? 32 * (E < 4 ? 4 : E > 16 ? 16 : E) : 128;
    if (act_bf16)
        NG_LAUNCH((moe_router_sigmoid_kernel<__nv_bfloat16>), n_rows, threads, smem, stream, (const __nv_bfloat16*)x, wr, corr,
                  wsg, weights, H, E, ldw, top_k, n_groups, keep_groups, softmax_scores, group_max, route_scale, n_identity);
    else
        NG_LAUNCH((moe_router_sigmoid_kernel<float>), n_rows, threads, smem, stream, (const float*)x, wr, corr, wsg, weights, H,
                  E, ldw, top_k, n_groups, keep_groups, softmax_scores, group_max, route_scale, n_identity);
    return ng_launch_status();
}

// moe_clamped_glu_scaled: out[row, c] = g' sigmoid(alpha g') (u' + 1) * weight, g' = min(g, limit), u' = clamp(u, -limit, limit),
//   g = gate_up[row, c], u = gate_up[row, I + c].  Columns below E*ff belong to expert c / ff: limit_e, weight
//   weights[row, c / ff]; the columns behind them to a shared expert: limit_s, weight weights[row, E] when `shared_gated`,
//   else 1.  Float32 until the one rounding of the result.
template <typename T>
__global__ void moe_clamped_glu_scaled_kernel(const T* __restrict__ gate_up, const float* __restrict__ weights, int ldw,
                                              T* __restrict__ out, int I, int E, int ff, float limit_e, float limit_s,
                                              float alpha, int shared_gated) {
    ng_pdl_trigger();
    ng_pdl_wait();
    const int row = blockIdx.y;
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= I) return;
    const bool routed = c < E * ff;
    const float limit = routed ? limit_e : limit_s;
    const float g = fminf(ng_ld(gate_up + (size_t)row * 2 * I + c), limit);
    const float u = fminf(fmaxf(ng_ld(gate_up + (size_t)row * 2 * I + I + c), -limit), limit);
    const float w = routed ? weights[(size_t)row * ldw + c / ff] : (shared_gated ? weights[(size_t)row * ldw + E] : 1.f);
    ng_st(out + (size_t)row * I + c, g / (1.f + expf(-alpha * g)) * (u + 1.f) * w);
}

NG_EXPORT int ng_moe_clamped_glu_scaled(const void* gate_up, const float* weights, int ldw, void* out, int n_rows, int I,
                                        int E, int ff, float limit_e, float limit_s, float alpha, int shared_gated,
                                        int act_bf16, cudaStream_t stream) {
    if (n_rows <= 0) return NG_OK;
    if (E <= 0 || ff <= 0 || I < E * ff || n_rows > 65535 || ldw < E + (shared_gated ? 1 : 0)) return NG_BAD_SIZE;
    dim3 grid((I + 255) / 256, n_rows);
    if (act_bf16)
        NG_LAUNCH((moe_clamped_glu_scaled_kernel<__nv_bfloat16>), grid, 256, 0, stream, (const __nv_bfloat16*)gate_up, weights,
                  ldw, (__nv_bfloat16*)out, I, E, ff, limit_e, limit_s, alpha, shared_gated);
    else
        NG_LAUNCH((moe_clamped_glu_scaled_kernel<float>), grid, 256, 0, stream, (const float*)gate_up, weights, ldw,
                  (float*)out, I, E, ff, limit_e, limit_s, alpha, shared_gated);
    return ng_launch_status();
}

// moe_identity_add: y[row, c] += weights[row] * x[row, c] with `weights` rows ldw apart (the column of the identity experts),
//   x of the activation type; y is float32 (the stream, or a partial sum) or of the activation type.
template <typename T, typename TY>
__global__ void moe_identity_add_kernel(TY* __restrict__ y, const T* __restrict__ x, const float* __restrict__ weights, int ldw, int H) {
    ng_pdl_trigger();
    ng_pdl_wait();
    const int row = blockIdx.y;
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= H) return;
    TY* p = y + (size_t)row * H + c;
    ng_st(p, fmaf(weights[(size_t)row * ldw], ng_ld(x + (size_t)row * H + c), ng_ld(p)));
}

NG_EXPORT int ng_moe_identity_add(void* y, const void* x, const float* weights, int ldw, int n_rows, int H, int y_f32, int act_bf16,
                                  cudaStream_t stream) {
    if (n_rows <= 0) return NG_OK;
    if (H <= 0 || ldw < 1 || n_rows > 65535) return NG_BAD_SIZE;
    dim3 grid((H + 255) / 256, n_rows);
    if (act_bf16 && y_f32)
        NG_LAUNCH((moe_identity_add_kernel<__nv_bfloat16, float>), grid, 256, 0, stream, (float*)y, (const __nv_bfloat16*)x, weights, ldw, H);
    else if (act_bf16)
        NG_LAUNCH((moe_identity_add_kernel<__nv_bfloat16, __nv_bfloat16>), grid, 256, 0, stream, (__nv_bfloat16*)y,
                  (const __nv_bfloat16*)x, weights, ldw, H);
    else
        NG_LAUNCH((moe_identity_add_kernel<float, float>), grid, 256, 0, stream, (float*)y, (const float*)x, weights, ldw, H);
    return ng_launch_status();
}
