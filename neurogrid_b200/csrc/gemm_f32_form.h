// Which form of the 32-bit product a size takes (gemm_f32.cu).  Plain C++.  Every form gives the same bits.
#pragma once

#define GF_CHUNK 64
#define GF_GROUP (16 * GF_CHUNK)                 // k of a group
#define GF_MAX_CLUSTER 8                         // groups that can be blocks of a cluster; a longer K walks its groups in one block
#define GR_COLS 8                                // few rows: columns of a block

static inline int gf_groups(int K) { return (K + GF_GROUP - 1) / GF_GROUP; }
static inline int gf_rows_of_block(int M) { return M <= 2 ? M : M <= 4 ? 4 : 8; }

// Few rows: whether the groups are the blocks of a cluster, or walked by one block, which has the next two on their way.  A
// block of one or two rows that walks has 75 to 125 KB in flight, and two of them an SM (of eight rows one) keep the memory as
// busy as a cluster does; so the cluster pays where the blocks alone leave SMs idle, or where they are more than fit at once.
// us with a small kernel that reads and writes the operands between two products, a cluster / one block:
//   1 row    1,024 x 2,048 5.3 / 5.0, 3,072 x 2,048 10.4 / 7.4, 16,384 x 2,048 35.8 / 29.9; 1,024 x 3,072 8.7 / 8.2, 2,048 x
//            3,072 10.8 / 7.8, 3,072 x 3,072 12.0 / 13.5; 1,024 x 4,608 6.9 / 10.2, 1,536 x 6,912 15.9 / 16.5, 2,048 x 8,192
//            19.5 / 18.6, 4,096 x 8,192 34.1 / 36.4
//   2 rows   512 x 1,536 4.8 / 5.0, 2,048 x 2,048 7.4 / 6.5, 3,072 x 1,536 10.4 / 10.0, 4,800 x 2,048 12.9 / 15.8, 6,144 x 2,048
//            19.6 / 18.9, 9,216 x 1,536 22.3 / 21.5, 16,384 x 2,048 37.6 / 40.1; three groups and more: 1,024 x 3,072 7.0 / 7.4, 2,048 x 4,608 13.7 / 22.0
//   4 rows   512 x 1,536 5.6 / 5.8, 1,536 x 1,536 7.5 / 7.0, 3,072 x 2,048 12.3 / 13.0; 2,048 x 4,608 18.8 / 26.0
//   8 rows   512 x 1,536 6.9 / 7.2, 1,024 x 1,536 8.4 / 7.5, 1,536 x 1,536 8.9 / 13.5; 2,048 x 4,608 26.4 / 33.5
//   24 rows  256 x 2,048 7.7 / 8.9; 32 rows 256 x 2,048 8.8 / 9.4, 3,072 x 2,048 47.1 / 79.4, 16,384 x 2,048 228 / 402
static inline bool gf_rows_cluster(int M, int N, int K) {
    const int groups = gf_groups(K), mr = gf_rows_of_block(M);
    if (groups < 2 || groups > GF_MAX_CLUSTER) return false;
    const long long blocks = (long long)((N + GR_COLS - 1) / GR_COLS) * ((M + mr - 1) / mr);
    if (mr == 1) return groups > 2 && ((groups > 3 && blocks <= 192) || blocks > 2 * 148);
    if (groups > 2) return true;
    if (blocks <= 96) return true;
    // two rows: a short second group is not worth a block; of the others, where the blocks' last wave would be nearly empty (296
    // a wave: 4,800 columns) or the waves are many
    if (mr == 2) return K - GF_GROUP > GF_GROUP / 2 && ((blocks > 512 && blocks <= 640) || blocks > 1024);
    return blocks > (mr == 4 ? 2 : 1) * 148;                             // more than are resident at once
}

// More rows: whether a tile's groups are the blocks of a cluster.  They are where one block a tile leaves SMs idle, or (296 tiles
// of 64 x 64 are resident at once) where a second wave would be nearly empty; a group that is half empty is worth less.
// us, mean over four surroundings of the product, a cluster / one block, 64 x 64 tiles of as many blocks as stand in brackets:
//   K = 1,280  [32] 51 / 51, [128] 83 / 68, [512] 259 / 182          K = 1,536  [48] 53 / 69, [72] 62 / 63, [96] 76 / 68 (96 rows of 3,072: 59 / 73), [576] 282 / 203
//   K = 2,048  [144] 77 / 120, [192] 115 / 139, [256] 152 / 145, [288] 146 / 139, [320] 184 / 209, [768] 383 / 394, [1,024] 496 / 471
//   K = 3,072  [192] 186 / 208, [256] 222 / 206, [320] 273 / 311, [512] 419 / 404          K = 4,608  [160] 224 / 314, [256] 352 / 317
//   K = 6,912  [144] 296 / 394, [240] 480 / 468, [384] 753 / 714     K = 8,192  [192] 440 / 552, [320] 708 / 834, [512] 1,112 / 1,093
static inline long long gf_tiles(int bm, int bn, int M, int N) { return (long long)((M + bm - 1) / bm) * ((N + bn - 1) / bn); }
static inline bool gf_tile_cluster(int M, int N, int K) {
    const int groups = gf_groups(K);
    if (groups < 2 || groups > GF_MAX_CLUSTER || K < GF_GROUP + GF_GROUP / 2) return false;
    if (K < 2 * GF_GROUP) return gf_tiles(32, 64, M, N) <= 2 * 72;
    const long long tiles = gf_tiles(64, 64, M, N);
    return tiles <= 200 || (tiles > 2 * 148 && tiles <= (groups == 2 ? 800 : 340));
}
// The tile: 0 for 64 x 64, 1 for 32 x 64, 2 for 32 x 32.  Large ones do more per byte of shared memory, but there must be enough of
// them.  us, mean over four surroundings, K = 1,024:
//   32 x 64 / 32 x 32, blocks of 32 x 64 in brackets  64 rows of 1,024 columns [32] 29 / 26, 64 of 2,048 [64] 35 / 31, 256 of 512 [64]
//       36 / 48, 128 of 1,024 [64] 30 / 34, 96 of 1,536 [72] 30 / 40, 192 of 1,024 [96] 46 / 66, 128 of 2,048 [128] 45 / 58 (256 of 1,024 [128] 59 / 46)
//   64 x 64 / 32 x 64, blocks of 64 x 64 in brackets  160 of 1,024 [48] 47 / 43, 256 of 1,536 [96] 53 / 47, 1,024 of
//       1,024 [256] 78 / 81, 192 of 9,216 [432] 110 / 110; K = 1,536: 640 of 1,536 [240] 109 / 121, 96 of 9,216 [288, half of them half empty] 105 / 87
static inline int gf_tile_size(int M, int N, int K) {
    const bool cluster = gf_tile_cluster(M, N, K);
    const long long s = cluster ? gf_groups(K) : 1, large = gf_tiles(64, 64, M, N);
    if (large * s >= 2 * 148 || (!cluster && large >= 200 && (M - 1) % 64 >= 32)) return 0;
    return gf_tiles(32, 64, M, N) * s >= (cluster || gf_groups(K) == 1 ? 64 : 72) ? 1 : 2;     // (a walk of 64: 280 / 239)
}
