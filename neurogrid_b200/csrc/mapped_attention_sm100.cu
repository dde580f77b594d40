// The attention of mapped_attention.cu for long bfloat16 portions on the Blackwell tensor cores: keys of 64, values of 64 or
// 128, one or two score maps a head, a window that keeps the first tokens, a soft cap.
//
// Same mathematics as the other kernels: q.k is a float32 sum of exact products, softmax and weights are float32; a weight
// enters the weighted sum as three bfloat16 terms hi + mid + lo (what is left is below 2^-24 of it), whose products with the
// bfloat16 values the tensor cores add in float32.
//
// A block runs two streams of 128 query rows of one head: with one map two row tiles that share keys and values, with two maps
// the two maps of one row tile (their own q and k, shared values), combined in the epilogue.  Warps:
//   warps 0-7, 8-15 softmax of stream 0 and 1: two threads a row (TMEM lane), 32 of a tile's keys each
//   warp 16         producer: TMA loads of Q and of the tiles' keys and values, gathered page by page (a lane per page)
//   warp 17 (, 18)  MMA issuer: S = Q K^T, O += P V (one elected lane), accumulators in TMEM; one a stream where S has two
//                   buffers (a stream does not wait behind the other's softmax), one for both otherwise (which keeps
//                   them out of step: two issuers took 125 us where one takes 106)
// TMEM of a stream: 64 columns of S, which the hi and mid terms of P replace, 32 of the lo terms, the values' columns of O.  The
// kernel is bound by the chain S - softmax - P V of its few warps, so with values of 64 S and P have two buffers, which fill
// the 512 columns, and the next tile's scores are there when a softmax warp comes for them.  Values of 128 leave room for one:
// there "S of tile j is there" also says that P V of the tile before has read its P and that O holds it (the tensor pipe
// runs the MMAs in order), and the streams fill each other's waits.  Every mbarrier wait is bounded; a waiter that gives up sets a status bit and the block runs to
// its end (TMEM is always released).  2,048 tokens, window 1,024: 32 heads of 64 with one map 67 us (212 us with
// the mma.sync kernel; 98 with one thread a row, one buffer and one issuer, 85 with two buffers, 77 with two threads a row), 16
// heads with two maps and values of 128 106 us (398 us; 114 with one thread a row).
#include "sm100_common.cuh"

#define HD 64                  // key size
#define BQ 128                 // query rows of a stream
#define BK 64                  // keys per tile
#define NG_STATUS_MAPPED_TIMEOUT 16
#define HK (BK / 2)            // keys of a softmax thread
#define PRODUCER 16            // the warps behind the sixteen of the softmax
#define ISSUER 17
static_assert(BQ == BLOCK_W, "a stream's query rows are the 128 rows of the MMA");

template <int M, int DV>
struct Cfg {
    static constexpr int NB = DV == 64 ? 2 : 1;                      // buffers of S and P a stream
    static constexpr int ISSUERS = NB;                               // warps that issue MMAs
    static constexpr int THREADS = 32 * (17 + ISSUERS);
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

// 32 consecutive float32 columns of this thread's TMEM lane, one load and one wait
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float (&v)[32]) {
    uint32_t r[32];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n\ttcgen05.wait::ld.sync.aligned;"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
                 : "r"(taddr) : "memory");
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}
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
__global__ void __launch_bounds__(Cfg<M, DV>::THREADS, 1)
mapped_attention_sm100_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                              const __grid_constant__ CUtensorMap map_v, const Params p) {
    typedef Cfg<M, DV> C;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* base = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    bf16* q_s = reinterpret_cast<bf16*>(base);                        // [2][BQ * HD], K-major swizzled
    bf16* kv_s = q_s + 2 * BQ * HD;                                   // [STAGES][STAGE_EL]
    int* pages = reinterpret_cast<int*>(kv_s + (size_t)C::STAGES * C::STAGE_EL);
    __shared__ uint64_t q_full, kv_full[C::STAGES], kv_empty[C::STAGES], s_full[2][C::NB], p_full[2][C::NB], o_ready[2][2], o_full;
    __shared__ uint32_t tmem_base;
    __shared__ float max_x[2][2][2][BQ], sum_x[2][2][BQ];             // what the two threads of a row tell each other
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
        for (int s = 0; s < C::STAGES; ++s) { mbar_init(&kv_full[s], 1); mbar_init(&kv_empty[s], C::ISSUERS == 2 ? streams : 1); }
        for (int s = 0; s < 2; ++s) {
            for (int b = 0; b < C::NB; ++b) { mbar_init(&s_full[s][b], 1); mbar_init(&p_full[s][b], 8); }
            for (int b = 0; b < 2; ++b) mbar_init(&o_ready[s][b], 1);
        }
        mbar_init(&o_full, C::ISSUERS == 2 ? streams : 1);
        hole = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == ISSUER) {
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
    for (int i = threadIdx.x; i < n_pages; i += C::THREADS) {
        const int page = trow[first_page + i], begin = (first_page + i) << p.ps_log2;
        if (tab_smem) pages[i] = page;
        if (no_page(page) && (begin + (1 << p.ps_log2) > lo_key || begin < p.keep_first)) hole = 1;
    }
    for (int i = threadIdx.x; (i << p.ps_log2) < min(p.keep_first, n_sink * BK); i += C::THREADS)
        if (no_page(trow[i])) hole = 1;
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    const uint32_t tmem = tmem_base;
    // columns: S and lo of every buffer of both streams, then both O
    auto tm_s = [&](int s, int b) { return tmem + (s * C::NB + b) * (BK + BK / 2); };
    auto tm_o = [&](int s) { return tmem + 2 * C::NB * (BK + BK / 2) + s * DV; };
    bool ok = true;

    if (warp == PRODUCER) {
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
    } else if (warp >= ISSUER) {
        // ------------------------------------------------------------------ MMA issuer
        // All lanes run the loop and its waits, one elected lane issues (descriptors stay in uniform registers)
        constexpr uint32_t idesc_s = make_idesc(BK, 0), idesc_o = make_idesc(DV, 1);
        ok = __all_sync(0xffffffffu, mbar_wait(&q_full, 0));
        const int s_lo = C::ISSUERS == 2 ? warp - ISSUER : 0, s_hi = C::ISSUERS == 2 ? s_lo : streams - 1;    // the warp's streams
        int n_s[2] = {0, 0}, n_p[2] = {0, 0};                         // tiles whose S / whose P V has been issued
        auto issue_s = [&](int s, int t) {                                   // S of tile t, over a P that an MMA issued before has read
            if (!__all_sync(0xffffffffu, mbar_wait(&kv_full[t % C::STAGES], (t / C::STAGES) & 1))) { ok = false; return; }
            tcgen05_fence_after();
            const uint64_t dq = make_desc_sw128(q_s + s * BQ * HD);
            const uint64_t dk = make_desc_sw128(kv_s + (size_t)(t % C::STAGES) * C::STAGE_EL + (M == 2 ? s * BK * HD : 0));
            const int b = n_s[s] % C::NB;
            const uint32_t ts = tm_s(s, b);
            if (leader) {
#pragma unroll
                for (int k = 0; k < HD / 16; ++k)
                    tcgen05_mma_f16(ts, dq + (uint64_t)(2 * k), dk + (uint64_t)(2 * k), idesc_s, k > 0);
                tcgen05_commit(&s_full[s][b]);
            }
            ++n_s[s];
            __syncwarp();
        };
        // Values that no row of the block sees (behind its last key, in front of the window, between the two) become zeros before
        // a product reads them: their weights are 0, and 0 times what another request left in a page may be NaN.  They lie in three
        // tiles at most.  This warp does it while it would wait for the softmax (in the softmax warps the same stores cost 2 to
        // 10 % of the kernel: registers).
        const int edge_kept = p.keep_first % BK ? n_sink - 1 : -1, edge_lo = lo_key % BK ? n_sink : -1;
        const int edge_last = pos_last % BK != BK - 1 ? n_tiles - 1 : -1;
        auto clear_unseen = [&](int t) {
            bf16* v = kv_s + (size_t)(t % C::STAGES) * C::STAGE_EL + M * BK * HD;
            for (int i = lane; i < BK * 8; i += 32) {                 // 128-byte rows whole: the swizzle stays inside
                const int k = i >> 3, key = tile_of(t) * BK + k;
                if (key <= pos_last && (key >= lo_key || key < p.keep_first)) continue;
#pragma unroll
                for (int c = 0; c < DV / 64; ++c) *reinterpret_cast<uint4*>(v + (c * BK + k) * 64 + (i & 7) * 8) = make_uint4(0u, 0u, 0u, 0u);
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
        };
        auto issue_pv = [&](int s, int t) {                                  // O += P V of tile t
            const int b = n_p[s] % C::NB;
            if (!__all_sync(0xffffffffu, mbar_wait(&p_full[s][b], (n_p[s] / C::NB) & 1))) { ok = false; return; }
            tcgen05_fence_after();
            // MN-major values: 64-column blocks BK * 64 elements apart, groups of eight keys 1,024 bytes apart
            const bf16* v = kv_s + (size_t)(t % C::STAGES) * C::STAGE_EL + M * BK * HD;
            uint64_t dv = make_desc_sw128_mn(v);
            dv = (dv & ~((uint64_t)0x3fff << 16)) | ((uint64_t)(BK * 64 * 2 >> 4) << 16);
            const uint32_t ts = tm_s(s, b), to = tm_o(s);
            const bool fresh = n_p[s] == 0;
            if (leader) {
#pragma unroll
                for (int term = 2; term >= 0; --term)                 // smallest terms first: lo (behind S), mid, hi
#pragma unroll
                    for (int k = 0; k < BK / 16; ++k)                 // 16 keys per MMA: 8 columns of P, 2,048 bytes of V
                        tcgen05_mma_f16_ts(to, ts + 32 * term + 8 * k, dv + (uint64_t)(128 * k), idesc_o,
                                           !(fresh && term == 2 && k == 0));
                if (C::NB == 2) tcgen05_commit(&o_ready[s][n_p[s] & 1]);
            }
            ++n_p[s];
            __syncwarp();
        };
        for (int t = 0; t <= n_tiles && ok && s_hi < streams; ++t) {
            // the values of tile t - 1 are there if S of the tile, which has been issued, was one of this warp's
            if ((t - 1 == edge_last || t - 1 == edge_lo || t - 1 == edge_kept) && t > 0 && (C::ISSUERS == 1 || sees(s_lo, t - 1))) clear_unseen(t - 1);
#pragma unroll
            for (int s = 0; s < 2; ++s) {
                if (s < s_lo || s > s_hi || !ok) continue;
                const bool pv = t > 0 && sees(s, t - 1), sk = t < n_tiles && sees(s, t);
                if (C::NB == 2 && sk) issue_s(s, t);                  // into the buffer whose P V was issued a round ago
                if (ok && pv) issue_pv(s, t - 1);
                if (ok && t > 0 && s == s_hi) {                       // the warp is done with the tile's keys and values
                    // (if it saw nothing of the tile: once the tile is there, so that its stage is not filled twice)
                    if (!pv) ok = __all_sync(0xffffffffu, mbar_wait(&kv_full[(t - 1) % C::STAGES], ((t - 1) / C::STAGES) & 1));
                    if (leader && ok) {
                        tcgen05_commit(&kv_empty[(t - 1) % C::STAGES]);
                        if (t == n_tiles) tcgen05_commit(&o_full);    // the warp's part of O is complete
                    }
                    __syncwarp();
                }
                if (ok && C::NB == 1 && sk) issue_s(s, t);
            }
        }
        if (!ok && leader) atomicOr(p.status, NG_STATUS_MAPPED_TIMEOUT);
    } else {
        // ------------------------------------------------------------------ softmax: two threads a query row of their stream
        // A thread has 32 of a tile's keys and half of the values' columns of O.  A wait that runs out does not leave the
        // loop: the two warps of a row meet at barriers, as often as the tiles say.
        const int s = warp >> 3, half = (warp >> 2) & 1, r = (warp & 3) * 32 + lane;
        const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
        const int row = (M == 2 ? 0 : s * BQ) + r;                    // within the block
        const bool warp_live = (M == 2 ? 0 : s * BQ) + (warp & 3) * 32 < rows_here;
        const int pos = pos_first + min(row, rows_here - 1);          // rows past the portion mirror its last row
        const int w_first = pos_first + min((M == 2 ? 0 : s * BQ) + (warp & 3) * 32, rows_here - 1);
        const int w_last = min(pos_last, w_first + 31);
        const float scale2 = p.scale * 1.4426950408889634f, inv_cap = p.softcap > 0.f ? p.scale / p.softcap : 0.f;
        const float cap2 = p.softcap * 1.4426950408889634f;
        const uint32_t to = tm_o(s) + lane_base + half * (DV / 2);
        auto pair_meets = [&]() { asm volatile("bar.sync %0, 64;" ::"r"(1 + s * 4 + (warp & 3)) : "memory"); };
        // m is the reference point of the exponentials (base 2), the same in both threads of a row.  It follows the running
        // maximum lazily: only when a tile's maximum exceeds it by more than 2^8 is O rescaled; otherwise weights simply
        // reach 256.
        float m = -INFINITY, l = 0.f;
        int n = 0;                                                    // tiles seen so far
        for (int t = 0; t < n_tiles && s < streams; ++t) {
            if (!sees(s, t)) continue;
            const int b = n % C::NB;
            const uint32_t ts = tm_s(s, b) + lane_base;
            if (ok) ok = __all_sync(0xffffffffu, mbar_wait(&s_full[s][b], (n / C::NB) & 1));
            tcgen05_fence_after();
            if (warp_live) {
                const int key0 = tile_of(t) * BK, my0 = key0 + half * HK;
                float sc[HK];
                tmem_ld32(ts + half * HK, sc);
                if (p.softcap > 0.f) {
#pragma unroll
                    for (int i = 0; i < HK; ++i) sc[i] = cap2 * tanh_ex2(sc[i] * inv_cap);
                } else {
#pragma unroll
                    for (int i = 0; i < HK; ++i) sc[i] *= scale2;
                }
                // only tiles that cross a row's diagonal or the window's edge need the mask
                const bool whole = key0 + BK - 1 <= w_first && (p.window <= 0 || key0 > w_last - p.window || key0 + BK <= p.keep_first);
                if (!whole || hole) {                                         // (a key without a page is not seen)
#pragma unroll
                    for (int i = 0; i < HK; ++i) {
                        const int key = my0 + i;
                        const bool vis = key <= pos && (p.window <= 0 || key > pos - p.window || key < p.keep_first);
                        sc[i] = vis && !(hole && no_page(trow[key >> p.ps_log2])) ? sc[i] : -INFINITY;
                    }
                }
                float m0 = sc[0], m1 = sc[1], m2 = sc[2], m3 = sc[3];
#pragma unroll
                for (int i = 4; i < HK; i += 4) {
                    m0 = fmaxf(m0, sc[i]);
                    m1 = fmaxf(m1, sc[i + 1]);
                    m2 = fmaxf(m2, sc[i + 2]);
                    m3 = fmaxf(m3, sc[i + 3]);
                }
                float mx = fmaxf(fmaxf(m0, m1), fmaxf(m2, m3));
                max_x[n & 1][s][half][r] = mx;
                tcgen05_fence_before();
                pair_meets();                                                 // the row's maximum; and both threads have read its S
                tcgen05_fence_after();
                mx = fmaxf(mx, max_x[n & 1][s][half ^ 1][r]);
                float corr = 1.f;
                if (mx > m + 8.f || (m == -INFINITY && mx > -INFINITY)) {     // move the reference point
                    corr = ex2(m - mx);                                       // 0 the first time
                    m = mx;
                }
                const float ref = m == -INFINITY ? 0.f : m;
                float l0 = 0.f, l1 = 0.f;
                uint32_t hi[HK / 2], mid[HK / 2], lo[HK / 2];
#pragma unroll
                for (int i = 0; i < HK / 2; ++i) {
                    const float a = ex2(sc[2 * i] - ref), c = ex2(sc[2 * i + 1] - ref);
                    l0 += a;
                    l1 += c;
                    hi[i] = pack_bf16(a, c);
                    const float ar = a - lo_f(hi[i]), cr = c - hi_f(hi[i]);
                    mid[i] = pack_bf16(ar, cr);
                    lo[i] = pack_bf16(ar - lo_f(mid[i]), cr - hi_f(mid[i]));
                }
                tmem_st16u(ts + half * (HK / 2), hi);                         // over the row's S
                tmem_st16u(ts + 32 + half * (HK / 2), mid);
                tmem_st16u(ts + 64 + half * (HK / 2), lo);
                l = l * corr + (l0 + l1);
                if (n > 0 && __any_sync(0xffffffffu, corr != 1.f)) {          // O has to hold the tiles before
                    if (C::NB == 2) {
                        if (ok) ok = __all_sync(0xffffffffu, mbar_wait(&o_ready[s][(n - 1) & 1], ((n - 1) >> 1) & 1));
                        tcgen05_fence_after();
                    }
#pragma unroll
                    for (int c = 0; c < DV / 2; c += 16) {
                        float v[16];
                        tmem_ld16(to + c, v);
#pragma unroll
                        for (int i = 0; i < 16; ++i) v[i] *= corr;
                        tmem_st16(to + c, v);
                    }
                }
                tmem_st_wait();
            }
            tcgen05_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&p_full[s][b]);
            ++n;
        }
        // ---- epilogue: O / l, the maps combined, the head's norm
        if (ok) ok = __all_sync(0xffffffffu, mbar_wait(&o_full, 0));
        if (!ok && lane == 0) atomicOr(p.status, NG_STATUS_MAPPED_TIMEOUT);
        tcgen05_fence_after();
        sum_x[s][half][r] = l;
        pair_meets();
        l += sum_x[s][half ^ 1][r];
        const float inv = l > 0.f ? 1.f / l : 0.f;
        const bool mine = ok && warp_live && s < streams;
        float* second = reinterpret_cast<float*>(kv_s) + (size_t)r * C::PITCH + half * (DV / 2);   // M == 2: the second map's rows, over the tiles
        if (M == 2) {
            if (s == 1 && mine) {
                const float f = -p.lambda * inv;
#pragma unroll
                for (int c = 0; c < DV / 2; c += 16) {
                    float v[16];
                    tmem_ld16(to + c, v);
#pragma unroll
                    for (int i = 0; i < 16; i += 4)
                        *reinterpret_cast<float4*>(second + c + i) = make_float4(v[i] * f, v[i + 1] * f, v[i + 2] * f, v[i + 3] * f);
                }
            }
            asm volatile("bar.sync 9, 512;" ::: "memory");            // the sixteen softmax warps
        }
        const bool writes = mine && (M == 1 || s == 0);
        float ss = 0.f;
        if (writes && (M == 2 || p.head_norm)) {
#pragma unroll
            for (int c = 0; c < DV / 2; c += 16) {
                float v[16];
                tmem_ld16(to + c, v);
#pragma unroll
                for (int i = 0; i < 16; i += 4) {
                    float4 a = make_float4(v[i] * inv, v[i + 1] * inv, v[i + 2] * inv, v[i + 3] * inv);
                    if (M == 2) {
                        const float4 d = *reinterpret_cast<const float4*>(second + c + i);
                        a.x += d.x; a.y += d.y; a.z += d.z; a.w += d.w;
                        *reinterpret_cast<float4*>(second + c + i) = a;
                    }
                    ss += (a.x * a.x + a.y * a.y) + (a.z * a.z + a.w * a.w);
                }
            }
        }
        max_x[0][s][half][r] = ss;
        pair_meets();
        ss = max_x[0][s][0][r] + max_x[0][s][1][r];
        if (writes) {
            float f = p.post_scale;
            if (p.head_norm) f *= rsqrtf(ss / (float)DV + p.eps);
            bf16* orow = p.out + (size_t)(q0 + r0 + row) * p.out_ld + (size_t)head * DV + half * (DV / 2);
#pragma unroll
            for (int c = 0; c < DV / 2; c += 16) {
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
    if (warp == ISSUER)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" :: "r"(tmem) : "memory");
}

template <int M, int DV>
static int launch(const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv, const Params& p, int n_entries, int max_q,
                  cudaStream_t stream) {
    constexpr int ROWS = M == 2 ? BQ : 2 * BQ;
    static std::atomic<unsigned long long> done{0};
    if (!ng_allow_smem(done, mapped_attention_sm100_kernel<M, DV>, (int)Cfg<M, DV>::smem())) return NG_LAUNCH_FAILED;
    const dim3 grid(p.nH, (max_q + ROWS - 1) / ROWS, n_entries);
    if (grid.y > 65535 || grid.z > 65535) return NG_BAD_SIZE;
    const size_t smem = Cfg<M, DV>::smem();
    const int threads = Cfg<M, DV>::THREADS;
    NG_LAUNCH((mapped_attention_sm100_kernel<M, DV>), grid, threads, smem, stream, mq, mk, mv, p);
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
