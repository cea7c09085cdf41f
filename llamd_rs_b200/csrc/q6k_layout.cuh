// The device layout of Q6_K weights ("T32") and the bit-level helpers that
// read it.
//
// A Q6_K block is 256 six-bit codes q, sixteen int8 scales and an f16 d
// (crates/llamd-quant/src/lib.rs:171-180). The reference's dot product keeps
// eight integer accumulators per block, one per residue r = element mod 8
// (crates/llamd-quant/src/dot.rs:175-188), and each accumulator sums
// scale[g] * (a[16g+r]*w[16g+r] + a[16g+8+r]*w[16g+8+r]) over the sixteen
// groups g. The layout below keeps the elements of a residue together, so that
// one thread produces those eight integers without a cross-lane reduction, and
// gives each of the four lanes that share a row of an integer MMA operand
// (q = lane % 4) a part of its own, so that the operand is made in registers:
//
//   residue r, weight n = 4j+k (j = word 0..7, k = byte 0..3)
//       <-> element e = 16*(2j + (k&1)) + 8*(k>>1) + r
//   byte value  W4 = ((q ^ 0x20) << 2)   i.e. 4*(q-32) as a signed byte
//   quad Q = 4*(r>>1) + (j&3) holds the four words i = 2*(r&1) + (j>>2): lane
//       q = j&3's words of residues 2(Q>>2) and 2(Q>>2)+1
//   its words W4_0..3 are stored in three: S_i = (W4_i & 0xFC..) | two bits of
//       W4_3 per byte (bits 7-6, 5-4, 3-2 for i = 0, 1, 2)
//
// so a block's codes take 16 quads x 3 words = 192 bytes, as in the file.
// 32 consecutive blocks form a 6720-byte tile: word-chunk c (16 B, c = 0..11)
// of block slot s sits at c*512 + 16*(s ^ (s>>3)), which makes every 16-byte
// load of a warp one contiguous 512-byte run and keeps the blocks of one column
// of an 8-blocks-a-row matrix in different shared-memory banks; then 32 x 16
// scale bytes, the four scales of q = 0, 1, 2, 3 one after the other; then 32 x 2
// bytes of d.
#pragma once
#include "common.cuh"

namespace llamd {

// 6-bit code of element e in a block in the reference's byte layout
// (crates/llamd-quant/src/lib.rs:198-222).
__host__ __device__ __forceinline__ uint32_t ggml_q6k_code(const uint8_t *blk, int e) {
    const int half = e >> 7, w = e & 127, c = w >> 5, l = w & 31;
    const uint8_t lo = blk[64 * half + l + 32 * (c & 1)];
    const uint32_t nib = (c >= 2) ? (uint32_t)(lo >> 4) : (uint32_t)(lo & 0x0F);
    const uint32_t hi = ((uint32_t)blk[128 + 32 * half + l] >> (2 * c)) & 3u;
    return nib | (hi << 4);
}

// element index of (residue r, word j, byte k)
__host__ __device__ __forceinline__ int t32_element(int r, int j, int k) {
    return 16 * (2 * j + (k & 1)) + 8 * (k >> 1) + r;
}

// place of (residue r, word j) among a block's 64 words: four times its quad, plus its word of the quad
__host__ __device__ __forceinline__ int t32_place(int r, int j) { return 16 * (r >> 1) + 4 * (j & 3) + 2 * (r & 1) + (j >> 2); }
// ... and back: the residue and the word at a place
__host__ __device__ __forceinline__ int t32_place_r(int place) { return 2 * (place >> 4) + ((place >> 1) & 1); }
__host__ __device__ __forceinline__ int t32_place_j(int place) { return ((place >> 2) & 3) + 4 * (place & 1); }
// place of a slot's 16 bytes in a run of 32, and of scale group g among a block's scale bytes
__host__ __device__ __forceinline__ int t32_slot(int slot) { return slot ^ (slot >> 3); }
__host__ __device__ __forceinline__ int t32_scale(int g) { return 4 * ((g >> 1) & 3) + 2 * (g >> 3) + (g & 1); }

// byte offset of code word wi (0..47) of block `unit` inside the tiled buffer
__host__ __device__ __forceinline__ size_t t32_word_offset(size_t unit, int wi) {
    const size_t tile = unit >> 5;
    return tile * kTileBytes + (size_t)(wi >> 2) * 512 + t32_slot((int)(unit & 31)) * 16 + (size_t)(wi & 3) * 4;
}
__host__ __device__ __forceinline__ size_t t32_scale_offset(size_t unit, int g) {
    return (unit >> 5) * kTileBytes + kTileScaleOff + t32_slot((int)(unit & 31)) * 16 + t32_scale(g);
}
__host__ __device__ __forceinline__ size_t t32_d_offset(size_t unit) {
    return (unit >> 5) * kTileBytes + kTileDOff + (unit & 31) * 2;
}

// q - 32 of element e of block `unit`, read back from the tiled buffer.
__device__ __forceinline__ int t32_weight(const uint8_t *tiled, size_t unit, int e) {
    const int r = e & 7, s = (e >> 3) & 1, g = e >> 4;
    const int place = t32_place(r, g >> 1), k = (s << 1) | (g & 1);
    const int quad = place >> 2, i = place & 3;
    uint32_t c6;
    if (i < 3) {
        c6 = (uint32_t)tiled[t32_word_offset(unit, 3 * quad + i) + k] >> 2;
    } else {
        const uint32_t b0 = tiled[t32_word_offset(unit, 3 * quad + 0) + k] & 3u;
        const uint32_t b1 = tiled[t32_word_offset(unit, 3 * quad + 1) + k] & 3u;
        const uint32_t b2 = tiled[t32_word_offset(unit, 3 * quad + 2) + k] & 3u;
        c6 = (b0 << 4) | (b1 << 2) | b2;
    }
    return (int)(c6 ^ 0x20u) - 32;
}

// Unpack the four W4 words of a quad from the three stored words.
__device__ __forceinline__ void unpack_quad(uint32_t s0, uint32_t s1, uint32_t s2, uint32_t w[4]) {
    w[0] = s0 & 0xFCFCFCFCu;
    w[1] = s1 & 0xFCFCFCFCu;
    w[2] = s2 & 0xFCFCFCFCu;
    const uint32_t u = ((s0 << 6) & 0xC0C0C0C0u) | ((s1 << 4) & 0x30303030u);
    w[3] = u | ((s2 << 2) & 0x0C0C0C0Cu);
}

// Q8_0 device layout: tiles of 32 rows x 1 block (1088 B): two 16-byte halves
// of each row's 32 quants, lane-interleaved, then the 32 f16 scales.
constexpr int kQ80TileBytes = 32 * 34;
__host__ __device__ __forceinline__ size_t q80_tile_offset(size_t row, size_t b, size_t blocks) {
    return ((row >> 5) * blocks + b) * kQ80TileBytes;
}

}  // namespace llamd
