// The lines between two kernels that compute the same bits, as plain functions of sizes. Each stands where the times of its
// two sides cross; both are given beside it.
#pragma once

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

}  // namespace llamd
