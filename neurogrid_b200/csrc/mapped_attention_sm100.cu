// The attention of mapped_attention.cu for long bfloat16 portions on the Blackwell tensor cores: keys of 64, values of 64 or
// 128, one or two score maps a head, a window that keeps the first tokens, a soft cap.
//
// Same mathematics as the other kernels: q.k is a float32 sum of exact products, softmax and weights are float32; a weight
// enters the weighted sum as three bfloat16 terms hi + mid + lo (what is left is below 2^-24 of it), whose products with the
// bfloat16 values the tensor cores add in float32.
//
// A block runs two streams of 128 query rows of one head: with one map two row tiles that share keys and values, with two maps
// the two maps of one row tile (their own q and k, shared values), combined in the epilogue.  Ten warps:
//   warps 0-3, 4-7  softmax of stream 0 and 1: thread r owns row r = TMEM lane r
//   warp 8          producer: TMA loads of Q and of the tiles' keys and values, gathered page by page (a lane per page)
//   warp 9          MMA issuer: S = Q K^T, O += P V (one elected lane), accumulators in TMEM
// TMEM of a stream: 64 columns of S, which the hi and mid terms of P replace, 32 of the lo terms, the values' columns of O.  The tensor
// pipe runs the MMAs in order: "S of tile j is there" says that P V of the tile before has read its P and that O holds it,
// so S has one buffer a stream and the streams fill each other's waits (while one stream's scores are on their way the
// other's softmax has the SM).  Every mbarrier wait is bounded; a waiter that gives up sets a status bit and the block runs to
// its end (TMEM is always released).  2,048 tokens, window 1,024, inside a step: 32 heads of 64 with one map 103 us (217 us with
// the mma.sync kernel), 16 heads with two maps and values of 128 120 us (406 us).
#include "sm100_common.cuh"

#define HD 64                  // key size
#define BQ 128                 // query rows of a stream
#define BK 64                  // keys per tile
#define NG_STATUS_MAPPED_TIMEOUT 16
#define THREADS 320
static_assert(BQ == BLOCK_W, "a stream's query rows are the 128 rows of the MMA");

template <int M, int DV>
struct Cfg {
    static constexpr int STAGES = M == 2 && DV == 128 ? 4 : 5;
    static constexpr int STAGE_EL = M * BK * HD + BK * DV;           // keys of every map, then values in blocks of 64 columns
    static constexpr int TABLE_INTS = 1024;
    static constexpr int PITCH = DV + 4;                             // floats of a row of the second map's part (epilogue)
    static constexpr size_t tiles() { return (size_t)STAGES * STAGE_EL * sizeof(bf16); }
    static_assert((size_t)BQ * PITCH * sizeof(float) <= (size_t)STAGES * STAGE_EL * sizeof(bf16), "the epilogue's rows fit over the tiles");
    static constexpr size_t smem() { return 2 * BQ * HD * sizeof(bf16) + tiles() + TABLE_INTS * sizeof(int) + 1024; }
};

struct Params {
    bf16* out;
    const int* table;
    const int* cu_q;
    const int* ctx_before;
    int* status;
    int out_ld, table_stride, nH, nG, ps_log2, num_pages, window, keep_first, head_norm;
    float scale, softcap, lambda, post_scale, eps;
};

__device__ __forceinline__ void tmem_st16u(uint32_t taddr, const uint32_t (&v)[16]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
                 :: "r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]),
                    "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]) : "memory");
}
// tanh(x) = 1 - 2 / (1 + e^(2x)): exact limits at both ends, absolute error of a few 1e-7
__device__ __forceinline__ float tanh_ex2(float x) { return 1.f - __fdividef(2.f, 1.f + ex2(x * 2.8853900817779268f)); }
__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ float lo_f(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float hi_f(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }

template <int M, int DV>
__global__ void __launch_bounds__(THREADS, 1)
mapped_attention_sm100_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                              const __grid_constant__ CUtensorMap map_v, const Params p) {
    typedef Cfg<M, DV> C;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* base = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    bf16* q_s = reinterpret_cast<bf16*>(base);                        // [2][BQ * HD], K-major swizzled
    bf16* kv_s = q_s + 2 * BQ * HD;                                   // [STAGES][STAGE_EL]
    int* pages = reinterpret_cast<int*>(kv_s + (size_t)C::STAGES * C::STAGE_EL);
    __shared__ uint64_t q_full, kv_full[C::STAGES], kv_empty[C::STAGES], s_full[2], p_full[2], o_full;
    __shared__ uint32_t tmem_base;
    __shared__ int hole;                                              // a key that rows of the block see has no page
    ng_pdl_trigger();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int e = blockIdx.z, head = blockIdx.x;
    uint32_t elected;                                                 // one lane of each warp, the same one every time it is asked
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.b32 %0, 1, 0, p;\n\t}" : "=r"(elected));
    const bool leader = elected != 0;
    constexpr int ROWS = M == 2 ? BQ : 2 * BQ;                        // rows of a block
    const int q0 = p.cu_q[e], qlen = p.cu_q[e + 1] - q0;
    const int r0 = (gridDim.y - 1 - blockIdx.y) * ROWS;               // heads fastest, the row tiles with the most keys first
    if (r0 >= qlen) {
        ng_pdl_wait();
        return;
    }
    const int ctx = p.ctx_before[e];
    const int g = head / (p.nH / p.nG);
    const int rows_here = min(ROWS, qlen - r0);
    const int streams = M == 2 || rows_here > BQ ? 2 : 1;
    const int pos_first = ctx + r0, pos_last = pos_first + rows_here - 1;
    // tiles of the block: those of the kept first tokens in front of the window, then the window's.  Entry t of that list is
    // tile `tile_of(t)`.
    const int lo_key = p.window > 0 ? max(0, pos_first - p.window + 1) : 0;      // the first key any row sees, but for kept ones
    const int lo_tile = lo_key / BK, hi_tile = pos_last / BK;
    const int n_sink = min((p.keep_first + BK - 1) / BK, lo_tile);
    const int n_tiles = n_sink + hi_tile - lo_tile + 1;
    auto tile_of = [&](int t) { return t < n_sink ? t : lo_tile + t - n_sink; };
    // whether a stream's rows see anything of a tile (every tile is seen by some stream: row tiles follow one another)
    auto sees = [&](int s, int t) {
        if (M == 2) return true;
        const int key0 = tile_of(t) * BK, first = pos_first + s * BQ, last = min(pos_last, first + BQ - 1);
        return key0 <= last && (p.window <= 0 || key0 + BK - 1 > first - p.window || key0 < p.keep_first);
    };

    if (threadIdx.x == 0) {
        mbar_init(&q_full, 1);
        for (int s = 0; s < C::STAGES; ++s) { mbar_init(&kv_full[s], 1); mbar_init(&kv_empty[s], 1); }
        for (int s = 0; s < 2; ++s) { mbar_init(&s_full[s], 1); mbar_init(&p_full[s], 4); }
        mbar_init(&o_full, 1);
        hole = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 9) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" :: "r"(smem_u32(&tmem_base)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    ng_pdl_wait();                                                    // q, the pages and the table are this step's data
    const int* trow = p.table + (size_t)e * p.table_stride;
    // page ids of the window's keys; those of kept tokens in front of it, or of a window too long for the buffer, are read where they are needed
    const int first_page = (lo_tile * BK) >> p.ps_log2;
    const int n_pages = (pos_last >> p.ps_log2) - first_page + 1;
    const bool tab_smem = n_pages <= C::TABLE_INTS;
    auto no_page = [&](int page) { return page < 0 || page >= p.num_pages; };
    __syncthreads();                                                  // `hole` is set
    for (int i = threadIdx.x; i < n_pages; i += THREADS) {
        const int page = trow[first_page + i], begin = (first_page + i) << p.ps_log2;
        if (tab_smem) pages[i] = page;
        if (no_page(page) && (begin + (1 << p.ps_log2) > lo_key || begin < p.keep_first)) hole = 1;
    }
    for (int i = threadIdx.x; (i << p.ps_log2) < min(p.keep_first, n_sink * BK); i += THREADS)
        if (no_page(trow[i])) hole = 1;
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    const uint32_t tmem = tmem_base;
    // columns: S and lo of both streams, then both O
    auto tm_s = [&](int s) { return tmem + s * (BK + BK / 2); };
    auto tm_o = [&](int s) { return tmem + 2 * (BK + BK / 2) + s * DV; };
    bool ok = true;

    if (warp == 8) {
        // ------------------------------------------------------------------ producer
        if (lane == 0) {
            mbar_expect_tx(&q_full, streams * BQ * HD * 2);
            for (int s = 0; s < streams; ++s)
                tma_load_2d(q_s + s * BQ * HD, &map_q, &q_full, (M == 2 ? head * 2 + s : head) * HD, q0 + r0 + (M == 2 ? 0 : s * BQ));
        }
        const int ps = 1 << p.ps_log2;
        const int oob_k = p.num_pages * p.nG * M * ps, oob_v = p.num_pages * p.nG * ps;       // out-of-range rows: TMA fills zeros
        for (int t = 0; t < n_tiles; ++t) {
            const int s = t % C::STAGES;
            ok = __all_sync(0xffffffffu, mbar_wait(&kv_empty[s], ((t / C::STAGES) & 1) ^ 1));
            if (!ok) break;
            bf16* st = kv_s + (size_t)s * C::STAGE_EL;
            if (lane == 0) mbar_expect_tx(&kv_full[s], C::STAGE_EL * 2);
            __syncwarp();
            const int c = lane << p.ps_log2;                          // one box per page (a tile is 64 / ps pages)
            if (c < BK) {
                const int key = tile_of(t) * BK + c;
                int page = -1;
                if (key <= pos_last) page = tab_smem && t >= n_sink ? pages[(key >> p.ps_log2) - first_page] : trow[key >> p.ps_log2];
                const bool there = !no_page(page);
#pragma unroll
                for (int m = 0; m < M; ++m)
                    tma_load_2d(st + m * BK * HD + c * HD, &map_k, &kv_full[s], 0, there ? ((page * p.nG + g) * M + m) * ps : oob_k);
#pragma unroll
                for (int b = 0; b < DV / 64; ++b)
                    tma_load_2d(st + M * BK * HD + b * BK * 64 + c * 64, &map_v, &kv_full[s], b * 64, there ? (page * p.nG + g) * ps : oob_v);
            }
        }
        if (!ok && lane == 0) atomicOr(p.status, NG_STATUS_MAPPED_TIMEOUT);
    } else if (warp == 9) {
        // ------------------------------------------------------------------ MMA issuer
        // All lanes run the loop and its waits, one elected lane issues (descriptors stay in uniform registers)
        constexpr uint32_t idesc_s = make_idesc(BK, 0), idesc_o = make_idesc(DV, 1);
        ok = __all_sync(0xffffffffu, mbar_wait(&q_full, 0));
        int p_phase[2] = {0, 0};
        bool begun[2] = {false, false};
        for (int t = 0; t <= n_tiles && ok; ++t) {
#pragma unroll
            for (int s = 0; s < 2; ++s) {
                if (s >= streams || !ok) break;
                if (t > 0 && sees(s, t - 1)) {                        // O += P V of the tile before
                    ok = __all_sync(0xffffffffu, mbar_wait(&p_full[s], p_phase[s]));
                    if (!ok) break;
                    p_phase[s] ^= 1;
                    tcgen05_fence_after();
                    // MN-major values: 64-column blocks BK * 64 elements apart, groups of eight keys 1,024 bytes apart
                    const bf16* v = kv_s + (size_t)((t - 1) % C::STAGES) * C::STAGE_EL + M * BK * HD;
                    uint64_t dv = make_desc_sw128_mn(v);
                    dv = (dv & ~((uint64_t)0x3fff << 16)) | ((uint64_t)(BK * 64 * 2 >> 4) << 16);
                    const uint32_t ts = tm_s(s), to = tm_o(s);
                    const bool fresh = !begun[s];
                    if (leader) {
#pragma unroll
                        for (int term = 2; term >= 0; --term)             // smallest terms first: lo (behind S), mid, hi
#pragma unroll
                            for (int k = 0; k < BK / 16; ++k)             // 16 keys per MMA: 8 columns of P, 2,048 bytes of V
                                tcgen05_mma_f16_ts(to, ts + 32 * term + 8 * k, dv + (uint64_t)(128 * k), idesc_o,
                                                   !(fresh && term == 2 && k == 0));
                    }
                    begun[s] = true;
                    __syncwarp();
                }
                if (t > 0 && s == streams - 1) {                      // the tile's keys and values may be overwritten
                    if (leader) {
                        tcgen05_commit(&kv_empty[(t - 1) % C::STAGES]);
                        if (t == n_tiles) tcgen05_commit(&o_full);    // O of both streams is complete
                    }
                    __syncwarp();
                }
                if (t < n_tiles && sees(s, t)) {                      // S of this tile, over the P that the MMAs above read
                    ok = __all_sync(0xffffffffu, mbar_wait(&kv_full[t % C::STAGES], (t / C::STAGES) & 1));
                    if (!ok) break;
                    tcgen05_fence_after();
                    const uint64_t dq = make_desc_sw128(q_s + s * BQ * HD);
                    const uint64_t dk = make_desc_sw128(kv_s + (size_t)(t % C::STAGES) * C::STAGE_EL + (M == 2 ? s * BK * HD : 0));
                    const uint32_t ts = tm_s(s);
                    if (leader) {
#pragma unroll
                        for (int k = 0; k < HD / 16; ++k)
                            tcgen05_mma_f16(ts, dq + (uint64_t)(2 * k), dk + (uint64_t)(2 * k), idesc_s, k > 0);
                        tcgen05_commit(&s_full[s]);
                    }
                    __syncwarp();
                }
            }
        }
        if (!ok && leader) atomicOr(p.status, NG_STATUS_MAPPED_TIMEOUT);
    } else {
        // ------------------------------------------------------------------ softmax: thread = query row of its stream
        const int s = warp >> 2, r = (warp & 3) * 32 + lane;
        const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
        const int row = (M == 2 ? 0 : s * BQ) + r;                    // within the block
        const bool warp_live = (M == 2 ? 0 : s * BQ) + (warp & 3) * 32 < rows_here;
        const int pos = pos_first + min(row, rows_here - 1);          // rows past the portion mirror its last row
        const int w_first = pos_first + min((M == 2 ? 0 : s * BQ) + (warp & 3) * 32, rows_here - 1);
        const int w_last = min(pos_last, w_first + 31);
        const float scale2 = p.scale * 1.4426950408889634f, inv_cap = p.softcap > 0.f ? p.scale / p.softcap : 0.f;
        const float cap2 = p.softcap * 1.4426950408889634f;
        const uint32_t ts = tm_s(s) + lane_base, to = tm_o(s) + lane_base;
        // m is the reference point of the exponentials (base 2).  It follows the running maximum lazily: only when a
        // tile's maximum exceeds it by more than 2^8 is O rescaled; otherwise weights simply reach 256.
        float m = -INFINITY, l = 0.f;
        int phase = 0;
        bool begun = false;
        for (int t = 0; t < n_tiles && s < streams; ++t) {
            if (!sees(s, t)) continue;
            ok = __all_sync(0xffffffffu, mbar_wait(&s_full[s], phase));
            if (!ok) break;
            phase ^= 1;
            tcgen05_fence_after();
            if (warp_live) {
                const int key0 = tile_of(t) * BK;
                float sc[BK];
                tmem_ld64(ts, sc);
                if (p.softcap > 0.f) {
#pragma unroll
                    for (int i = 0; i < BK; ++i) sc[i] = cap2 * tanh_ex2(sc[i] * inv_cap);
                } else {
#pragma unroll
                    for (int i = 0; i < BK; ++i) sc[i] *= scale2;
                }
                // only tiles that cross a row's diagonal or the window's edge need the mask
                const bool whole = key0 + BK - 1 <= w_first && (p.window <= 0 || key0 > w_last - p.window || key0 + BK <= p.keep_first);
                if (!whole || hole) {                                         // (a key without a page is not seen)
#pragma unroll
                    for (int i = 0; i < BK; ++i) {
                        const int key = key0 + i;
                        const bool vis = key <= pos && (p.window <= 0 || key > pos - p.window || key < p.keep_first);
                        sc[i] = vis && !(hole && no_page(trow[key >> p.ps_log2])) ? sc[i] : -INFINITY;
                    }
                }
                float m0 = sc[0], m1 = sc[1], m2 = sc[2], m3 = sc[3];
#pragma unroll
                for (int i = 4; i < BK; i += 4) {
                    m0 = fmaxf(m0, sc[i]);
                    m1 = fmaxf(m1, sc[i + 1]);
                    m2 = fmaxf(m2, sc[i + 2]);
                    m3 = fmaxf(m3, sc[i + 3]);
                }
                const float mx = fmaxf(fmaxf(m0, m1), fmaxf(m2, m3));
                float corr = 1.f;
                if (mx > m + 8.f || (m == -INFINITY && mx > -INFINITY)) {     // move the reference point
                    corr = ex2(m - mx);                                       // 0 the first time
                    m = mx;
                }
                const float ref = m == -INFINITY ? 0.f : m;
                float l0 = 0.f, l1 = 0.f;
#pragma unroll
                for (int h = 0; h < BK; h += 32) {                            // 32 keys at a time: 16 words of each term
                    uint32_t hi[16], mid[16], lo[16];
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        const float a = ex2(sc[h + 2 * i] - ref), b = ex2(sc[h + 2 * i + 1] - ref);
                        l0 += a;
                        l1 += b;
                        hi[i] = pack_bf16(a, b);
                        const float ar = a - lo_f(hi[i]), br = b - hi_f(hi[i]);
                        mid[i] = pack_bf16(ar, br);
                        lo[i] = pack_bf16(ar - lo_f(mid[i]), br - hi_f(mid[i]));
                    }
                    // over this row's S (all of it has been read)
                    tmem_st16u(ts + h / 2, hi);
                    tmem_st16u(ts + 32 + h / 2, mid);
                    tmem_st16u(ts + 64 + h / 2, lo);
                }
                l = l * corr + (l0 + l1);
                if (begun && __any_sync(0xffffffffu, corr != 1.f)) {          // O holds the tiles before (S of this one is behind them)
#pragma unroll
                    for (int c = 0; c < DV; c += 16) {
                        float v[16];
                        tmem_ld16(to + c, v);
#pragma unroll
                        for (int i = 0; i < 16; ++i) v[i] *= corr;
                        tmem_st16(to + c, v);
                    }
                }
                begun = true;
                tmem_st_wait();
            }
            tcgen05_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&p_full[s]);
        }
        // ---- epilogue: O / l, the maps combined, the head's norm
        if (ok) ok = __all_sync(0xffffffffu, mbar_wait(&o_full, 0));
        if (!ok && lane == 0) atomicOr(p.status, NG_STATUS_MAPPED_TIMEOUT);
        tcgen05_fence_after();
        const float inv = l > 0.f ? 1.f / l : 0.f;
        float* second = reinterpret_cast<float*>(kv_s) + (size_t)r * C::PITCH;       // M == 2: the second map's rows, over the tiles
        if (M == 2) {
            if (s == 1 && warp_live && ok) {
                const float f = -p.lambda * inv;
#pragma unroll
                for (int c = 0; c < DV; c += 16) {
                    float v[16];
                    tmem_ld16(to + c, v);
#pragma unroll
                    for (int i = 0; i < 16; i += 4)
                        *reinterpret_cast<float4*>(second + c + i) = make_float4(v[i] * f, v[i + 1] * f, v[i + 2] * f, v[i + 3] * f);
                }
            }
            asm volatile("bar.sync 1, 256;" ::: "memory");            // the eight softmax warps
        }
        if (ok && warp_live && (M == 1 || s == 0) && s < streams) {
            float ss = 0.f;
            if (M == 2 || p.head_norm) {
#pragma unroll
                for (int c = 0; c < DV; c += 16) {
                    float v[16];
                    tmem_ld16(to + c, v);
#pragma unroll
                    for (int i = 0; i < 16; i += 4) {
                        float4 a = make_float4(v[i] * inv, v[i + 1] * inv, v[i + 2] * inv, v[i + 3] * inv);
                        if (M == 2) {
                            const float4 b = *reinterpret_cast<const float4*>(second + c + i);
                            a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w;
                            *reinterpret_cast<float4*>(second + c + i) = a;
                        }
                        ss += (a.x * a.x + a.y * a.y) + (a.z * a.z + a.w * a.w);
                    }
                }
            }
            float f = p.post_scale;
            if (p.head_norm) f *= rsqrtf(ss / (float)DV + p.eps);
            bf16* orow = p.out + (size_t)(q0 + r0 + row) * p.out_ld + (size_t)head * DV;
#pragma unroll
            for (int c = 0; c < DV; c += 16) {
                float v[16];
                if (M == 2) {
#pragma unroll
                    for (int i = 0; i < 16; i += 4) {
                        const float4 a = *reinterpret_cast<const float4*>(second + c + i);
                        v[i] = a.x; v[i + 1] = a.y; v[i + 2] = a.z; v[i + 3] = a.w;
                    }
                } else {
                    tmem_ld16(to + c, v);
#pragma unroll
                    for (int i = 0; i < 16; ++i) v[i] *= inv;
                }
                uint32_t w[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) w[i] = pack_bf16(v[2 * i] * f, v[2 * i + 1] * f);
                if (row < rows_here) {
                    *reinterpret_cast<uint4*>(orow + c) = make_uint4(w[0], w[1], w[2], w[3]);
                    *reinterpret_cast<uint4*>(orow + c + 8) = make_uint4(w[4], w[5], w[6], w[7]);
                }
            }
        }
    }
    tcgen05_fence_before();
    __syncthreads();
    if (warp == 9)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" :: "r"(tmem) : "memory");
}

template <int M, int DV>
static int launch(const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv, const Params& p, int n_entries, int max_q,
                  cudaStream_t stream) {
    constexpr int ROWS = M == 2 ? BQ : 2 * BQ;
    static bool attr = false;
    if (!attr) {
        if (cudaFuncSetAttribute(mapped_attention_sm100_kernel<M, DV>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)Cfg<M, DV>::smem()) != cudaSuccess)
            return NG_LAUNCH_FAILED;
        attr = true;
    }
    const dim3 grid(p.nH, (max_q + ROWS - 1) / ROWS, n_entries);
    if (grid.y > 65535 || grid.z > 65535) return NG_BAD_SIZE;
    const size_t smem = Cfg<M, DV>::smem();
    NG_LAUNCH((mapped_attention_sm100_kernel<M, DV>), grid, THREADS, smem, stream, mq, mk, mv, p);
    return ng_launch_status();
}

// q [n_rows, nH * n_maps * 64] bfloat16; keys [P, nG * n_maps, page, 64]; values [P, nG, page, dv]; out rows out_ld apart (a
// multiple of 8).  Rows are named by cu_q and ctx_before, as for the other kernels.
NG_EXPORT int ng_mapped_attention_sm100(const void* q, const void* k_pages, const void* v_pages, const int* table,
                                        int table_stride, const int* cu_q, const int* ctx_before, void* out, int out_ld, int n_rows,
                                        int n_entries, int max_q, int nH, int nG, int n_maps, int d, int dv, int page_size,
                                        int num_pages, int window, int keep_first, float scale, float softcap, float lambda,
                                        float post_scale, float eps, int head_norm, int* status, cudaStream_t stream) {
    if (n_entries <= 0 || max_q <= 0 || n_rows <= 0) return NG_OK;
    if (d != HD || (dv != 64 && dv != 128) || n_maps < 1 || n_maps > 2 || page_size < 8 || page_size > 64 ||
        (page_size & (page_size - 1)) || nH <= 0 || nG <= 0 || nH % nG || window < 0 || keep_first < 0 ||
        out_ld < nH * dv || out_ld % 8 || !status || (((uintptr_t)q | (uintptr_t)k_pages | (uintptr_t)v_pages | (uintptr_t)out) & 15))
        return NG_BAD_SIZE;
    int ps_log2 = 0;
    while ((1 << ps_log2) < page_size) ++ps_log2;
    CUtensorMap mq, mk, mv;
    if (!tensor_map(q, n_rows, nH * n_maps * HD, BQ, &mq) ||
        !tensor_map(k_pages, (long long)num_pages * nG * n_maps * page_size, HD, page_size, &mk) ||
        !tensor_map(v_pages, (long long)num_pages * nG * page_size, dv, page_size, &mv))
        return NG_LAUNCH_FAILED;
    const Params p{(bf16*)out, table, cu_q, ctx_before, status, out_ld, table_stride, nH, nG, ps_log2, num_pages, window, keep_first,
                   head_norm, scale, softcap, lambda, post_scale, eps};
    if (n_maps == 1) return dv == 64 ? launch<1, 64>(mq, mk, mv, p, n_entries, max_q, stream) : launch<1, 128>(mq, mk, mv, p, n_entries, max_q, stream);
    return dv == 64 ? launch<2, 64>(mq, mk, mv, p, n_entries, max_q, stream) : launch<2, 128>(mq, mk, mv, p, n_entries, max_q, stream);
}
