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
    // two rows: a short second group is not worth a block; of the others, where the blocks' last round would be nearly empty (296
    // a round: 4,800 columns) or the rounds are many
    if (mr == 2) return K - GF_GROUP > GF_GROUP / 2 && ((blocks > 512 && blocks <= 640) || blocks > 1024);
    return blocks > (mr == 4 ? 2 : 1) * 148;                             // more than are resident at once
}
