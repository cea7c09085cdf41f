// The lines between two kernels that compute the same bits, as plain functions of sizes. Each stands where the times of its
// two sides cross; both are given beside it.
#pragma once
#include <stddef.h>

namespace llamd {

// From here on the experts of a pass run as a grouped GEMM over the scatter plan instead of a matvec per (token, expert): the
// GEMM folds an expert's weights once for all its tokens, the matvec repeats its integer work for each. So the line is in (token,
// expert) pairs: 1.65 per expert, and what the plan and the GEMM's launches cost on top, which weighs less the larger an expert is.
// weights: n_embd * n_ff_expert. us a layer of a decode pass, matvec / GEMM, by experts (used per token) of width x n_embd:
//   8 (2) x 1536 x 2048:   8 tokens 87.5 / 93.9, 10: 96.2 / 96.8, 12: 109.7 / 105.2, 24: 146.5 / 113.8
//   8 (2) x 3072 x 4096:   6: 180.5 / 184.6, 8: 193.2 / 193.0, 12: 260.8 / 214.7, 32: 506.5 / 250.4
//   16 (2) x 256 x 2048:  16: 81.0 / 84.1, 24: 90.0 / 90.0, 32: 96.2 / 93.1, 56: 122.8 / 113.5
//   32 (4) x 768 x 2048:  16: 124.4 / 127.4, 18: 133.2 / 134.7, 20: 139.2 / 134.4, 32: 172.4 / 144.7
//   64 (6) x 1536 x 2048: 18: 240.2 / 248.3, 20: 257.1 / 254.5, 24: 288.5 / 266.9, 56: 565.3 / 312.8
//   128 (8) x 256 x 2048: 32: 142.8 / 149.0, 36: 159.6 / 160.5, 40: 168.6 / 165.6, 56: 203.8 / 179.9
//   128 (8) x 768 x 2048: 24: 215.6 / 233.7, 28: 240.0 / 242.1, 32: 262.1 / 249.8, 64: 452.8 / 300.6
//   256 (8) x 512 x 2048: 32: 209.9 / 252.2, 56: 325.9 / 335.1, 64: 354.3 / 341.2
//   512 (10) x 512 x 2048: 26: 225.8 / 312.5, 51: 372.8 / 458.8, 64: 430.1 / 491.9
inline bool experts_on_gemm(long long pairs, int n_expert, long long weights) {
    return 20 * pairs >= 33LL * n_expert + (4LL * n_expert + 220) * (768 * 2048) / weights;
}

// Softmax and weighted values of one kv head's query heads (attn_out_gqa_kernel): four CTAs to an SM, with half the products ahead of
// a chain, or three. Four wins only where four are there: where the launch has more than three and a half to an SM and their
// shared memory lets them (smem bytes each and the 1 KB that the system takes, of 228 KB: rows of up to 768 positions).
// us a layer, three / four, batches of 128: rows of 288 positions 311.4 / 307.5, 700: 425.8 / 419.5, 768: 442.0 / 435.5, 1000: 499.6 /
// 499.7, 1500: 647.2 / 653.3, 2500: 913.7 / 926.7. Batches of 32 (512 CTAs): 133.2 / 132.0 to 171.9 / 171.5; 48: 161.5 / 162.1 to 216.7 / 216.6;
// a 48-layer pass of 32 behind 72 to 264 positions 11985 / 12016.
// Tiles of 37 tokens (592) behind 300 positions 164.9 / 161.0, 700: 0.980 times, 800: 208.6 / 209.0, 4000: 571.9 / 588.6.
inline bool attn_out_four_ctas(long long ctas, size_t smem) { return 2 * ctas > 7 * 148 && 4 * (smem + 1024) <= 228 * 1024; }

// Attention of a small tile of one sequence by kv head (attention_small_tile), or by the tiled kernels. positions: a row of its
// scores; ctas: of its second launch, 16 a token for four kv heads. Rows of more than 4352 positions leave one CTA to an SM, and those
// that wait for another's end lose more than the tiled kernels' emptier tiles. us a layer, tiled / by kv head, f32 cache:
//   behind 4360 positions: 9 tokens (144 CTAs) 312 / 214, 10: 315 / 314, 14: 328 / 341, 19: 337 / 445, 24: 340 / 468, 56 behind 4500: 455 / 995
//   behind 5300:           9: 360 / 239, 10: 362 / 358, 14: 375 / 391, 19: 385 / 511, 24: 388 / 543, 56: 508 / 1137
// Beyond 5376 positions the rows do not fit.
inline bool small_tile_by_kv_head(int positions, long long ctas) { return positions <= 4352 || (positions <= 5376 && ctas <= 148); }

// A host-facing Q6_K product of several sequences on the integer GEMM, which folds a weight once for all of them, or by matvec. Up to
// eight blocks a row from three sequences on: four CTAs of 16 rows share an SM there and a wave of them is as short as the matvec.
// Wider rows leave room for two CTAs, beyond 16 blocks for one, so a matrix of few rows is one wave of long chains, and the line is
// the matvec's work against the GEMM's waves. us of quantizing and product, matvec / GEMM (launches come in ticks of 2 us):
//   rows x blocks   2 sequences      3              4              6              8
//   2048 x 8         7.8 / 7.7     8.1 / 7.6      8.3 / 7.5      8.3 / 7.7      8.3 / 8.3
//   151936 x 8      81.9 / 87.1  141.4 / 88.0   176.0 / 88.1   238.2 / 88.2   301.9 / 90.1
//   3072 x 12        9.7 / 9.8     8.3 / 9.9     10.3 / 9.7     14.4 / 9.9     16.4 / 10.3
//   512 x 16         8.2 / 8.3     7.5 / 8.3      8.2 / 8.3      8.2 / 8.3      8.2 / 8.3
//   2048 x 16        8.2 / 8.3     8.3 / 8.3     10.2 / 9.1     12.3 / 10.1    14.4 / 10.2
//   1024 x 20        8.3 / 10.3    8.2 / 10.3    10.3 / 10.3    10.3 / 10.3    14.4 / 10.3
//   512 x 24         8.3 / 10.3    8.0 / 10.3     8.3 / 10.3    10.3 / 10.3    10.3 / 10.3
//   3072 x 24       12.4 / 16.4   14.4 / 16.4    18.8 / 16.4    24.6 / 17.3    30.4 / 17.5
//   5120 x 24       15.0 / 22.6   20.5 / 22.6    24.6 / 23.5    34.9 / 24.4    44.2 / 24.6
//   10000 x 24      24.6 / 36.0   41.0 / 36.4    50.8 / 36.9    69.7 / 36.9   102.5 / 36.9
inline bool product_on_gemm(int blocks, int rows, int nseq) {
    if (nseq < 3 || blocks > 24) return false;
    if (blocks <= 8) return true;
    const long long per_sm = blocks <= 16 ? 2 : 1, tiles = (rows + 15LL) / 16, waves = (tiles + 148 * per_sm - 1) / (148 * per_sm);
    return (nseq + 1LL) * rows * blocks * per_sm >= 160000 * waves;
}

}  // namespace llamd
