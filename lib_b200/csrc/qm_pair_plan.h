// Which tile a matmul by CTA pairs (qm_gemm_pair.cu) runs with. Host code without a context: sizes in, plan out.
#pragma once
#include <math.h>
#include <stdint.h>

#include <algorithm>

// CTAs per tile (1 or 2), tokens per tile, K shares per tile (one cluster), and the tiles that the launch may meet.
struct QmPairPlan {
    int cg, bn, splitk;
    int64_t tiles;
};

// clusters[CTAs per tile - 1][K shares]: clusters of that size that the device runs at once.
typedef int QmPairClusters[2][5];

// A single matrix of `rows` rows with m tokens.
// Estimated cycles: a stage of 128 columns takes 4 cycles per token column on the tensor cores (a CTA alone also copies
// and reads all of B: 5), at least what its dequantization and hand-over take; a tile's accumulator read-out is hidden
// by the next tile only where two accumulators fit. The least is set at 500 cycles; time stamps inside the kernel put a
// stage of 160 tokens at about 725, with which the formula would take larger tiles for many tokens (256 instead of
// 160 for 2048 tokens of 4096 x 4096). Which is faster has not been timed.
inline QmPairPlan qm_plan_matmul(const QmPairClusters &clusters, int64_t rows, int64_t m, int units) {
    QmPairPlan best = {2, 64, 1, (rows + 255) / 256 * ((m + 63) / 64)};
    double best_cost = 0;
    for (int cg = 1; cg <= 2; cg++)
        for (int bn = 32; bn <= 256; bn += 32) {
            const int64_t tiles = (rows + 128 * cg - 1) / (128 * cg) * ((m + bn - 1) / bn);
            for (int s = 1; s * cg <= 4; s *= 2) {   // clusters of up to four CTAs (of eight only 15 fit at once)
                const int at_once = clusters[cg - 1][s];
                if (at_once < 1 || (s > 1 && (tiles > at_once || units < s))) continue;
                const int64_t rounds = (tiles + at_once - 1) / at_once;
                const double stage = std::max((cg == 2 ? 4.0 : 5.0) * bn, 500.0), readout = 12.0 * bn + (s > 1 ? 2000 : 0);
                const double cost = rounds * (units * 2.0 / s * stage + 500) + (bn <= 128 ? readout : rounds * readout);
                if (best_cost == 0 || cost < best_cost) {
                    best = {cg, bn, s, tiles};
                    best_cost = cost;
                }
            }
        }
    return best;
}

// Token tiles of bn that the experts' lists can make at most: no list is longer than `longest` and together they hold
// at most `rows` tokens. (A list of l tokens makes ceil(l / bn) <= (l + bn - 1) / bn tiles, none if it is empty.)
inline int64_t qm_grouped_token_tiles(int64_t longest, int64_t rows, int64_t experts, int64_t bn) {
    return std::min(experts * ((longest + bn - 1) / bn), (rows + std::min(experts, rows) * (bn - 1)) / bn);
}

// Tokens per tile for lists of l tokens: tiles of equal size, at most 160 (the tile of the layer that this was measured
// with, 8 experts and lists of 128 on average; an expert's weights are dequantized once per token tile, so lists of 161
// to 256 might gain from one larger tile: not timed).
inline int qm_grouped_bn(int64_t l) {
    const int64_t nt = (l + 159) / 160;
    return (int)std::max<int64_t>(32, ((l + nt - 1) / nt + 31) & ~(int64_t)31);
}

// The list length that a tile is chosen for where only the mean is known: two standard deviations of a random choice more.
inline int64_t qm_typical_list(int64_t rows, int64_t experts) {
    const double mean = (double)rows / experts;
    return (int64_t)std::max(1.0, mean + 2.0 * sqrt(mean));
}

// Grouped launch: `experts` matrices of out_cols output columns (with SwiGLU: gate rows) over token lists of at most
// `longest` tokens, `rows` together; tiles chosen for lists of `typical` tokens.
// Few experts (expert-parallel runs) leave pairs idle: two of them then share a tile's K. A K-shared launch starts a
// cluster per tile that the lists may hold, so it is taken only where all of those fit at once, and whether it may be is
// seen from the bound on the tiles, not from a mean list. MoE layers, shared -> not: 1 expert 4096 x 4096 of 128 tokens
// 61 -> 65 us, 2 experts 1024 x 4096 of 64 tokens 48 -> 52; where clusters stand in line for tiles that are mostly empty,
// 16 experts 512 x 2048 of 1024 pairs 138 -> 64 us, 4 experts 2048 x 4096 of 600 pairs 115 -> 83.
// Sharing K changes the order of additions. It is decided by share_longest and share_rows, which a caller that may know
// the lists or not gives as the bounds that hold in both cases, so that the bits do not depend on which.
inline QmPairPlan qm_plan_grouped(const QmPairClusters &clusters, int64_t out_cols, bool swiglu, int64_t longest,
                                  int64_t typical, int64_t rows, int experts, int units, bool may_share,
                                  int64_t share_longest, int64_t share_rows) {
    const int tile_rows = swiglu ? 128 : 256;
    const int64_t row_tiles = (out_cols + tile_rows - 1) / tile_rows;
    QmPairPlan p = {2, qm_grouped_bn(typical), 1, 0};
    p.tiles = row_tiles * qm_grouped_token_tiles(longest, rows, experts, p.bn);
    const int share_bn = qm_grouped_bn(qm_typical_list(share_rows, experts));
    if (may_share && !swiglu && units >= 2 &&
        row_tiles * qm_grouped_token_tiles(share_longest, share_rows, experts, share_bn) <= clusters[1][2])
        p.splitk = 2;
    return p;
}
