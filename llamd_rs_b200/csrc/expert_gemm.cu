// Q6_K x Q8_K for several tokens on the integer tensor path: the grouped expert
// matmuls of prompts, drafts and batches, and the dense projections and the
// output matrix of the same passes.
//
// The reference's arithmetic (crates/llamd-quant/src/dot.rs:138-196) keeps, per
// (row, token, block b, residue r = element mod 8), the integer
//     aux[r] = sum over 16 groups g, 2 elements s of  scale[g] * w[16g+8s+r] * a[16g+8s+r]
// and then accumulates in f32, in block order:  sums[r] += (f16(d_b) * ad_b) * (float)aux[r].
// That fixes the shape of the tensor-core formulation: each (b, r) is its own
// 32-deep contraction whose result needs its own f32 scaling, so the MMA is
//     D[16 rows x 8 tokens] = A[16 x 32] * B[32 x 8]     (mma.sync m16n8k32, s8 x s8 -> s32)
// with A = U = scale[g]*w folded per row and B = the token's Q8_K bytes of that
// residue. U needs 13 bits, so 4U is split exactly into its high byte (signed)
// and its low byte (unsigned): two MMAs, aux = 64*hi + lo/4. Integer results are
// exact in any order; the f32 tail runs in the reference's order, so the result
// is bit-identical to the scalar loop and to the dp4a matvec kernels.
// This mirrors the role of crates/llamd-vulkan/shaders/q6k_expert_cm.comp
// (cooperative-matrix s8 GEMM with f32 scaling per 16-K group).
//
// What it costs is instruction issue: the packed codes have to become operands (some 40 instructions per 512 weights and warp)
// and every 128 sums need 2 MMAs (10 cycles each, which keep the FP32 pipe from issuing) and 8 packed FP32 instructions.
// The operands are made in registers by the lane that multiplies with them -- the weight layout gives every lane its own words
// (q6k_layout.cuh) -- and used for all the token tiles at hand. Three forms (gemm_launch):
//   q6k_gemm_few_kernel     a warp folds all residues of its blocks: up to 16 tokens a group at up to three blocks a row, and up to 8
//                           tokens of one group (a projection, the head) at any number;
//   q6k_gemm_shared_kernel  groups of more than 40 tokens at up to four blocks a row (24 at two): rows folded into shared memory once for four
//                           warps;
//   q6k_gemm_kernel         everything else: four warps, a residue pair each, share 16 rows and up to 8 tiles.
// us for 128 experts, gate and up (2 x 768 x 2048) / down (2048 x 768), 8 experts per token, before (every row tile folded into
// shared memory, a warp per token tile) and now: 32 tokens 200 / 101, 114 / 58; 128: 243 / 119, 141 / 82; 512: 360 / 180, 257 / 164; 2048:
// 910 / 465, 795 / 465.
#include "packed_f32.cuh"
#include "q6k_layout.cuh"

namespace llamd {

constexpr int kGemmRows = 16;

struct GemmParams {
    const uint8_t *w[3];  // tiled Q6_K; up to three matrices that share the activations
    float *out[3];
    int rows[3];
    int tile_begin[3];    // first blockIdx.x of each matrix
    int njobs;
    int nb;               // blocks per row
    int row_tiles;        // row tiles per CTA
    int raw_bytes;        // shared memory for their blocks
    const uint32_t *aq_rm;  // activations in operand order (t32_place): [index][nb][64 words]
    const float *ad;        // [index][nb]
    // token groups: group e = pairs [gstart[e], gstart[e]+gcount[e]); pair p reads activation act_map[p] and writes
    // output row block out_map[p]. gstart == null: one group of n_tokens pairs, cut into runs of run_tiles token tiles
    // (blockIdx.y). maps == null: identity.
    const int32_t *gstart, *gcount, *act_map, *out_map;
    int n_tokens, run_tiles;
    long long expert_units;  // blocks between consecutive experts in w
    int prefetch_ahead;      // grouped: CTA i asks L2 for the weights of CTA i + prefetch_ahead (0: off)
    // expert parallelism: output row block o lives on GPU o / out_div, at local row block o % out_div (null: out[j])
    float *const *out_tab;
    int out_div;
    // copies of the matrices kept folded (null: fold from w): [expert][row tile] images of fold_tile_bytes (kImageBlockBytes)
    const uint8_t *folded[3];
    long long fold_tile_bytes;
    f32x2 one;  // kOne2
};

struct Quad { uint32_t v[4]; };
__device__ __forceinline__ void opaque(Quad &q, uint32_t c) {
#pragma unroll
    for (int i = 0; i < 4; i++) asm volatile("mov.u32 %0, %1;" : "=r"(q.v[i]) : "r"(c));
}
template <bool UNSIGNED>
__device__ __forceinline__ void mma_8(int (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1, const Quad &q) {
    if (UNSIGNED)
        asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};"
                     : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3])
                     : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "r"(q.v[0]), "r"(q.v[1]), "r"(q.v[2]), "r"(q.v[3]));
    else
        asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};"
                     : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3])
                     : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "r"(q.v[0]), "r"(q.v[1]), "r"(q.v[2]), "r"(q.v[3]));
}

__device__ __forceinline__ void copy_async16(uint32_t dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
// ... through L1: the CTAs of an SM read the same activations, and in L2 a few tokens' lines are too few for all SMs
__device__ __forceinline__ void copy_async16_l1(uint32_t dst, const void *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copy_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

__device__ __forceinline__ f32x2 add2x(f32x2 a, f32x2 b) {  // a + b where no product is an operand, see packed_f32.cuh
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

// Natural-order Q8_K quants -> operand order, one thread per word.
__global__ void q8k_residue_major_kernel(const int8_t *__restrict__ aq, uint32_t *__restrict__ rm, size_t nblocks) {
    pdl_trigger();
    pdl_wait();
    const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (i >= nblocks * 64) return;
    const size_t blk = i >> 6;
    const int r = t32_place_r((int)i & 63), j = t32_place_j((int)i & 63);
    const uint8_t *src = reinterpret_cast<const uint8_t *>(aq) + blk * 256;
    rm[i] = (uint32_t)src[t32_element(r, j, 0)] | ((uint32_t)src[t32_element(r, j, 1)] << 8) | ((uint32_t)src[t32_element(r, j, 2)] << 16) |
            ((uint32_t)src[t32_element(r, j, 3)] << 24);
}

__device__ __forceinline__ int job_of_tile(const GemmParams &p, int x) {
    int j = 0;
    if (p.njobs > 1 && x >= p.tile_begin[1]) j = 1;
    if (p.njobs > 2 && x >= p.tile_begin[2]) j = 2;
    return j;
}

// ---- the A operand: scale times weight, split into bytes ----
// Two weights of one scale group are folded by ONE 32-bit multiply-add: with q = w + 32 in [0, 63],
//     (4*q0 | 4*q2 << 16) * sc + (C | C << 16),  C = 32768 - 128*sc
// is, as an integer, sum_i (4*U_i + 32768) << 16i, and every term lies in [16384, 49152], so the two 16-bit fields hold
// 4*U_i + 32768 with no carry between them: the low byte is 4*(U & 63), the high byte (U >> 6) + 128.
struct Fold {
    uint32_t mask, sc[4], c[4];  // 0x00FC00FC; a lane's four scales of one row: groups 2q, 2q+1, 2q+8, 2q+9
};
__device__ __forceinline__ void fold_scales(Fold &f, uint32_t packed) {
    asm("mov.u32 %0, 0x00FC00FC;" : "=r"(f.mask));  // (in a register: a LOP3 takes one immediate)
#pragma unroll
    for (int i = 0; i < 4; i++) {
        f.sc[i] = (uint32_t)(int)(int8_t)(packed >> (8 * i));
        f.c[i] = f.sc[i] * (uint32_t)(-128 * 0x00010001) + 0x80008000u;
    }
}
__device__ __forceinline__ uint32_t and_xor(uint32_t a, uint32_t m, uint32_t x) {  // (a & m) ^ x; written out it becomes two instructions
    uint32_t r;
    asm("lop3.b32 %0, %1, %2, %3, 0x78;" : "=r"(r) : "r"(x), "r"(a), "r"(m));
    return r;
}
// A lane's words of one row and residue pair: s = the quad's three stored words. Operand registers `reg` and reg + 2 of both
// residues (words j = q and q + 4). Bytes 0 and 2 of a word share a scale, as do bytes 1 and 3.
__device__ __forceinline__ void fold_quad(const uint32_t (&s)[3], const Fold &f, int reg, uint32_t (&hi)[2][4], uint32_t (&lo)[2][4]) {
    // the fourth word's codes are the low bit pairs of the other three (what else is in it the mask takes away)
    const uint32_t w01 = ((s[0] << 6) & 0xC0C0C0C0u) | ((s[1] << 4) & ~0xC0C0C0C0u);
    const uint32_t w3 = (w01 & 0xF0F0F0F0u) | ((s[2] << 2) & ~0xF0F0F0F0u);
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const uint32_t w = i < 3 ? s[i < 3 ? i : 0] : w3;
        const int half = i & 1;
        const uint32_t ve = and_xor(w, f.mask, 0x00800080u) * f.sc[2 * half] + f.c[2 * half];
        const uint32_t vo = and_xor(w >> 8, f.mask, 0x00800080u) * f.sc[2 * half + 1] + f.c[2 * half + 1];
        hi[i >> 1][reg + 2 * half] = __byte_perm(ve, vo, 0x7351) ^ 0x80808080u;
        lo[i >> 1][reg + 2 * half] = __byte_perm(ve, vo, 0x6240);
    }
}

// The weights of the CTA that will take this one's place on the SM start their trip from HBM now.
template <bool FOLDED = false>
__device__ __forceinline__ void prefetch_ahead(const GemmParams &p, int ahead) {
    if (threadIdx.x || ahead <= 0) return;
    const long long lin = (long long)blockIdx.y * gridDim.x + blockIdx.x + ahead;
    const int px = (int)(lin % gridDim.x), pe = (int)(lin / gridDim.x), pj = job_of_tile(p, px);
    if (pe >= (int)gridDim.y || p.gcount[pe] <= 0) return;
    const int pt = (px - p.tile_begin[pj]) * p.row_tiles;
    const size_t u0 = (size_t)pe * (size_t)p.expert_units + (size_t)pt * kGemmRows * p.nb;
    const size_t a = u0 >> 5, z = (u0 + (size_t)min(p.row_tiles * kGemmRows, p.rows[pj] - pt * kGemmRows) * p.nb - 1) >> 5;
    const uint8_t *src = FOLDED ? p.folded[pj] + ((size_t)pe * ((p.rows[pj] + kGemmRows - 1) / kGemmRows) + pt) * (size_t)p.fold_tile_bytes
                                : p.w[pj] + a * kTileBytes;
    const uint32_t bytes = FOLDED ? (uint32_t)p.fold_tile_bytes : (uint32_t)((z - a + 1) * kTileBytes);
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(src), "r"(bytes) : "memory");
}

struct RowTile {
    int j, row0, live;   // matrix, first row, rows that exist (<= 16)
    uint32_t raw;        // shared-memory address of the tile that holds block `unit0` and the ones behind it, or of the image
    int unit0;           // block of (row0, 0), counted from that tile's first
};

// The operands of one block of a row tile, made by the lane that multiplies with them. u: block of the lane's row g4 + 8h,
// counted from the tile at `raw`.
__device__ __forceinline__ void fold_block(uint32_t raw, int u, int q4, const uint32_t (&word_off)[3], int h, uint32_t (&hi)[2][4],
                                           uint32_t (&lo)[2][4], float &d) {
    const uint32_t tile = raw + (uint32_t)(u >> 5) * kTileBytes, sl = (uint32_t)(u & 31), at = tile + 16u * (uint32_t)t32_slot((int)sl);
    uint32_t s[3], sc;
    uint16_t db;
#pragma unroll
    for (int i = 0; i < 3; i++) asm volatile("ld.shared.u32 %0, [%1];" : "=r"(s[i]) : "r"(at + word_off[i]));
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(sc) : "r"(at + kTileScaleOff + 4u * (uint32_t)q4));
    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(db) : "r"(tile + kTileDOff + 2u * sl));
    Fold f;
    fold_scales(f, sc);
    fold_quad(s, f, h, hi, lo);
    d = f16_bits_to_f32(db);
}
__device__ __forceinline__ void fold_offsets(int rp, int q4, uint32_t (&word_off)[3]) {
#pragma unroll
    for (int i = 0; i < 3; i++) word_off[i] = (uint32_t)((3 * rp + ((3 * q4 + i) >> 2)) * 512 + ((3 * q4 + i) & 3) * 4);
}
// The image of a folded row tile: [block][rp][hi of residue 2rp, of 2rp + 1, lo of both][lane] x 16 bytes, then the 16 x nb
// block scales as floats.
constexpr int kImageBlockBytes = 4 * 4 * 512;

// NT token tiles from tile0 on against one row tile: warp rp owns residues 2rp and 2rp + 1; their sums meet in shared memory at
// the end and are added in order.
template <int NT, int SLOTS, bool FOLDED>
__device__ __forceinline__ void team_tiles(const GemmParams &p, const RowTile &rt, int first, int count, int tile0, uint32_t s_ring, float *s_ring_f,
                                           float *s_ad, int ad_stride, int tid) {
    constexpr int D = SLOTS / NT;  // blocks of activations on their way
    const int nb = p.nb, rp = tid >> 5, lane = tid & 31, rows = p.rows[rt.j];
    const int g4 = lane >> 2, q4 = lane & 3, n0 = tile0 * 8;
    __syncthreads();  // (the ring and the scales of the tiles before are no longer read)
    auto act = [&](int tok) -> unsigned {
        const int pt = first + min(n0 + tok, count - 1);
        return p.act_map ? (unsigned)p.act_map[pt] : (unsigned)pt;
    };
    // A lane copies the 16 bytes that it will itself multiply with: word q4 and q4 + 4 of its residues, token g4 of the tile.
    const uint32_t ring = s_ring + (uint32_t)(rp * SLOTS * 512 + lane * 16);
    const uint4 *src[NT];
#pragma unroll
    for (int t = 0; t < NT; t++) src[t] = reinterpret_cast<const uint4 *>(p.aq_rm) + (size_t)act(t * 8 + g4) * nb * 16 + rp * 4 + q4;
    // (places without a token are left as they are: their sums go nowhere, and one line read by every lane of the GPU is slow)
    const bool last_live = n0 + (NT - 1) * 8 + g4 < count;
    auto request = [&](int b, int slot) {
        if (b < nb) {
#pragma unroll
            for (int t = 0; t < NT; t++)
                if (t + 1 < NT || last_live) copy_async16(ring + (uint32_t)((slot * NT + t) * 512), src[t] + (size_t)b * 16);
        }
        copy_commit();
    };
#pragma unroll
    for (int s = 0; s < D; s++) request(s, s);
    for (int i = tid; i < NT * 8 * nb; i += 128) {  // the tiles' activation scales, [block][token]
        const int tok = i / nb, b = i - tok * nb;
        s_ad[b * ad_stride + tok] = __ldg(p.ad + (size_t)act(tok) * nb + b);
    }
    f32x2 sum[NT][2][2];
#pragma unroll
    for (int t = 0; t < NT; t++) sum[t][0][0] = sum[t][0][1] = sum[t][1][0] = sum[t][1][1] = 0ull;
    // -(1.5 * 2^29 + 1.5 * 2^21), twice: see the tail
    const f32x2 one = p.one, off = 0xCE40C000CE40C000ull;
    const int u[2] = {rt.unit0 + min(g4, rt.live - 1) * nb, rt.unit0 + min(g4 + 8, rt.live - 1) * nb};
    uint32_t word_off[3];
    fold_offsets(rp, q4, word_off);
    Quad qh, ql;
    opaque(qh, 0x4E400000u);
    opaque(ql, 0x4A400000u);
    copy_wait<D>();  // the weights' copies came before the ring's
    __syncthreads();
    int slot = 0;
    for (int b = 0; b < nb; b++) {
        uint32_t hi[2][4], lo[2][4];
        f32x2 d[2];
        if (FOLDED) {
            const uint32_t at = rt.raw + (uint32_t)(b * kImageBlockBytes + rp * 2048 + lane * 16);
#pragma unroll
            for (int rr = 0; rr < 2; rr++) {
                asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(hi[rr][0]), "=r"(hi[rr][1]), "=r"(hi[rr][2]), "=r"(hi[rr][3]) : "r"(at + rr * 512));
                asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(lo[rr][0]), "=r"(lo[rr][1]), "=r"(lo[rr][2]), "=r"(lo[rr][3]) : "r"(at + 1024 + rr * 512));
            }
#pragma unroll
            for (int h = 0; h < 2; h++) {
                float df;
                asm volatile("ld.shared.f32 %0, [%1];" : "=f"(df) : "r"(rt.raw + (uint32_t)(nb * kImageBlockBytes + ((g4 + 8 * h) * nb + b) * 4)));
                d[h] = pack2(df, df);
            }
        } else {
#pragma unroll
            for (int h = 0; h < 2; h++) {
                float df;
                fold_block(rt.raw, u[h] + b, q4, word_off, h, hi, lo, df);
                d[h] = pack2(df, df);
            }
        }
        copy_wait<D - 1>();
#pragma unroll
        for (int t = 0; t < NT; t++) {
            uint32_t bw[4];
            asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(bw[0]), "=r"(bw[1]), "=r"(bw[2]), "=r"(bw[3])
                         : "r"(ring + (uint32_t)((slot * NT + t) * 512)));
            const f32x2 a = *reinterpret_cast<const f32x2 *>(s_ad + b * ad_stride + t * 8 + 2 * q4);
            const f32x2 dsc[2] = {mul2(d[0], a), mul2(d[1], a)};
#pragma unroll
            for (int rr = 0; rr < 2; rr++) {
                // The sums land on 1.5 * 2^29 (whose last place is 64) and on 1.5 * 2^21 (last place 1/4), so that they come
                // out as the floats 64*hi and lo/4 with that offset. Both differences below are exact: multiples of 64
                // below 2^25, and |aux| < 2^24.
                int ch[4], cl[4];
                mma_8<false>(ch, hi[rr], bw[2 * rr], bw[2 * rr + 1], qh);
                mma_8<true>(cl, lo[rr], bw[2 * rr], bw[2 * rr + 1], ql);
#pragma unroll
                for (int h = 0; h < 2; h++) {  // rows g4 and g4 + 8, tokens 2 q4 and 2 q4 + 1
                    const f32x2 x = add2x(pack2(__int_as_float(ch[2 * h]), __int_as_float(ch[2 * h + 1])), off);
                    const f32x2 aux = add2x(pack2(__int_as_float(cl[2 * h]), __int_as_float(cl[2 * h + 1])), x);
                    sum[t][rr][h] = add2(sum[t][rr][h], mul2(dsc[h], aux), one);
                }
            }
        }
        request(b + D, slot);
        slot = slot + 1 == D ? 0 : slot + 1;
    }
    // y = ((((((s0+s1)+s2)+s3)+s4)+s5)+s6)+s7, two tiles at a time: [7 terms][16 token places][16 rows] where the ring was
    float *s_x = s_ring_f;
#pragma unroll
    for (int t0 = 0; t0 < NT; t0 += 2) {
        __syncthreads();
#pragma unroll
        for (int t = t0; t < t0 + 2 && t < NT; t++) {
#pragma unroll
            for (int h = 0; h < 2; h++) {
                float *x = s_x + ((t - t0) * 8 + q4) * 16 + g4 + 8 * h;  // (token 2 q4 + e has place q4 + 4 e)
                if (rp == 0) {
                    const float2 v = unpack2(add2(sum[t][0][h], sum[t][1][h], one));
                    x[0] = v.x, x[4 * 16] = v.y;
                } else {
                    const float2 v = unpack2(sum[t][0][h]), w = unpack2(sum[t][1][h]);
                    x += (2 * rp - 1) * 256;
                    x[0] = v.x, x[4 * 16] = v.y, x[256] = w.x, x[256 + 4 * 16] = w.y;
                }
            }
        }
        __syncthreads();
#pragma unroll
        for (int t = t0; t < t0 + 2 && t < NT; t++) {
            const int row = tid & 15, place = tid >> 4;
            const float *x = s_x + ((t - t0) * 8 + place) * 16 + row;
            float y = x[0];
#pragma unroll
            for (int r = 1; r < 7; r++) y = __fadd_rn(y, x[r * 256]);
            const int n = n0 + t * 8 + 2 * (place & 3) + (place >> 2);
            if (n < count && row < rt.live) {
                long long o = p.out_map ? p.out_map[first + n] : first + n;
                float *out = p.out[rt.j];
                if (p.out_tab) {  // the rows of a pair go to the GPU the pair's token lives on (plain peer stores)
                    out = p.out_tab[o / p.out_div];
                    o %= p.out_div;
                }
                out[o * rows + rt.row0 + row] = y;
            }
        }
    }
}

// A lane's four outputs: rows g4 (ya) and g4 + 8 (yb) of the row tile, tokens n and n + 1 of the group.
__device__ __forceinline__ void store_pair(const GemmParams &p, int j, int row0, int live, int first, int count, int n, int g4, float2 ya, float2 yb) {
#pragma unroll
    for (int e = 0; e < 2; e++) {
        if (n + e >= count) continue;
        long long o = p.out_map ? p.out_map[first + n + e] : first + n + e;
        float *out = p.out[j];
        if (p.out_tab) {  // the rows of a pair go to the GPU the pair's token lives on (plain peer stores)
            out = p.out_tab[o / p.out_div];
            o %= p.out_div;
        }
        out += o * p.rows[j] + row0;
        if (g4 < live) out[g4] = e ? ya.y : ya.x;
        if (g4 + 8 < live) out[g4 + 8] = e ? yb.y : yb.x;
    }
}

// ---- few tokens per group ----
// Up to 8 NT tokens against one row tile, one warp per BW blocks of the rows: a warp folds all eight residues of its blocks, so
// that a block's scales, addresses and token scales are prepared once for eight residues and not for two. The products of the
// tail wait in registers; then the warps add theirs in block order, each to the sums that the warp before it left in shared
// memory, and the last one adds the eight residues. DIRECT (short rows): one warp has all the blocks of its own row tile, and
// takes one tile group after the other; otherwise there is one group of at most eight tokens.
// us, a residue pair per warp / this: the head for 8 tokens 95 / 86; down of 128 experts, 32 tokens 72 / 58, 128: 94 / 82. (Groups of 8
// blocks a row: no gain, 130 / 131 for gate and up of 64 tokens, the products' registers cost the occupancy.)
template <int NT>
struct Sums {
    f32x2 v[NT][8][2];  // [token tile][residue][rows g4, g4 + 8] x tokens 2 q4, 2 q4 + 1
};
template <int NT, int BW, bool DIRECT>
__device__ __forceinline__ void few_tiles(const GemmParams &p, const RowTile &rt, int first, int count, int tile0, uint32_t s_act, float *s_x, int w,
                                          int nw, int lane) {
    const int nb = p.nb;
    const int g4 = lane >> 2, q4 = lane & 3, n0 = tile0 * 8, b0 = w * BW;
    auto act = [&](int tok) -> unsigned {
        const int pt = first + min(n0 + tok, count - 1);
        return p.act_map ? (unsigned)p.act_map[pt] : (unsigned)pt;
    };
    // this warp's blocks of the tokens: a lane copies the 16 bytes per residue pair that it will itself multiply with
    const uint32_t mine = s_act + (uint32_t)(lane * 16);
    float ad[NT][2][BW];
#pragma unroll
    for (int t = 0; t < NT; t++) {
        const uint4 *src = reinterpret_cast<const uint4 *>(p.aq_rm) + ((size_t)act(t * 8 + g4) * nb + b0) * 16 + q4;
        if (n0 + t * 8 + g4 < count) {  // (places without a token are left as they are: their sums go nowhere)
#pragma unroll
            for (int i = 0; i < BW; i++)
                if (b0 + i < nb) {
#pragma unroll
                    for (int rp = 0; rp < 4; rp++) copy_async16_l1(mine + (uint32_t)(((t * BW + i) * 4 + rp) * 512), src + i * 16 + rp * 4);
                }
        }
#pragma unroll
        for (int e = 0; e < 2; e++) {
            const float *a = p.ad + (size_t)act(t * 8 + 2 * q4 + e) * nb + b0;
#pragma unroll
            for (int i = 0; i < BW; i++) ad[t][e][i] = __ldg(a + min(i, nb - 1 - b0));
        }
    }
    copy_commit();
    const f32x2 one = p.one, off = 0xCE40C000CE40C000ull;  // -(1.5 * 2^29 + 1.5 * 2^21), twice: see team_tiles
    const int u[2] = {rt.unit0 + min(g4, rt.live - 1) * nb + b0, rt.unit0 + min(g4 + 8, rt.live - 1) * nb + b0};
    uint32_t word_off[3];
    fold_offsets(0, q4, word_off);
    Quad qh, ql;
    opaque(qh, 0x4E400000u);
    opaque(ql, 0x4A400000u);
    copy_wait<0>();
    __syncthreads();  // everyone's pieces of the weights
    Sums<NT> sums, prod[DIRECT ? 1 : BW];
#pragma unroll
    for (int t = 0; t < NT; t++)
#pragma unroll
        for (int r = 0; r < 8; r++) sums.v[t][r][0] = sums.v[t][r][1] = 0ull;
#pragma unroll
    for (int i = 0; i < BW; i++) {
        if (b0 + i < nb) {
            uint32_t at[2];
            Fold f[2];
            f32x2 dsc[NT][2];
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const uint32_t tile = rt.raw + (uint32_t)((u[h] + i) >> 5) * kTileBytes, sl = (uint32_t)((u[h] + i) & 31);
                at[h] = tile + 16u * (uint32_t)t32_slot((int)sl);
                uint32_t sc;
                uint16_t db;
                asm volatile("ld.shared.u32 %0, [%1];" : "=r"(sc) : "r"(at[h] + kTileScaleOff + 4u * (uint32_t)q4));
                asm volatile("ld.shared.u16 %0, [%1];" : "=h"(db) : "r"(tile + kTileDOff + 2u * sl));
                fold_scales(f[h], sc);
                const float d = f16_bits_to_f32(db);
#pragma unroll
                for (int t = 0; t < NT; t++) dsc[t][h] = mul2(pack2(d, d), pack2(ad[t][0][i], ad[t][1][i]));
            }
#pragma unroll
            for (int rp = 0; rp < 4; rp++) {
                uint32_t hi[2][4], lo[2][4];
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    uint32_t s[3];
#pragma unroll
                    for (int c = 0; c < 3; c++) asm volatile("ld.shared.u32 %0, [%1];" : "=r"(s[c]) : "r"(at[h] + word_off[c] + (uint32_t)(rp * 1536)));
                    fold_quad(s, f[h], h, hi, lo);
                }
#pragma unroll
                for (int t = 0; t < NT; t++) {
                    uint32_t bw[4];
                    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(bw[0]), "=r"(bw[1]), "=r"(bw[2]), "=r"(bw[3])
                                 : "r"(mine + (uint32_t)(((t * BW + i) * 4 + rp) * 512)));
#pragma unroll
                    for (int rr = 0; rr < 2; rr++) {
                        int ch[4], cl[4];
                        mma_8<false>(ch, hi[rr], bw[2 * rr], bw[2 * rr + 1], qh);
                        mma_8<true>(cl, lo[rr], bw[2 * rr], bw[2 * rr + 1], ql);
#pragma unroll
                        for (int h = 0; h < 2; h++) {
                            const f32x2 x = add2x(pack2(__int_as_float(ch[2 * h]), __int_as_float(ch[2 * h + 1])), off);
                            const f32x2 y = mul2(dsc[t][h], add2x(pack2(__int_as_float(cl[2 * h]), __int_as_float(cl[2 * h + 1])), x));
                            if (DIRECT) sums.v[t][2 * rp + rr][h] = add2(sums.v[t][2 * rp + rr][h], y, one);
                            else prod[DIRECT ? 0 : i].v[t][2 * rp + rr][h] = y;
                        }
                    }
                }
            }
        }
    }
    f32x2 *x = reinterpret_cast<f32x2 *>(s_x) + lane;  // [token tile][residue][rows][lane]
    if (!DIRECT) {
        for (int ww = 0; ww < nw; ww++) {
            if (ww == w) {
                if (ww > 0) {
#pragma unroll
                    for (int k = 0; k < NT * 16; k++) sums.v[k >> 4][(k >> 1) & 7][k & 1] = x[k * 32];
                }
#pragma unroll
                for (int i = 0; i < BW; i++)
                    if (b0 + i < nb) {
#pragma unroll
                        for (int k = 0; k < NT * 16; k++)
                            sums.v[k >> 4][(k >> 1) & 7][k & 1] = add2(sums.v[k >> 4][(k >> 1) & 7][k & 1], prod[DIRECT ? 0 : i].v[k >> 4][(k >> 1) & 7][k & 1], one);
                    }
                if (ww + 1 < nw) {
#pragma unroll
                    for (int k = 0; k < NT * 16; k++) x[k * 32] = sums.v[k >> 4][(k >> 1) & 7][k & 1];
                }
            }
            if (ww + 1 < nw) __syncthreads();
        }
    }
    if (DIRECT || w == nw - 1) {
        // y = ((((((s0+s1)+s2)+s3)+s4)+s5)+s6)+s7
#pragma unroll
        for (int t = 0; t < NT; t++) {
            f32x2 y[2];
#pragma unroll
            for (int h = 0; h < 2; h++) {
                y[h] = sums.v[t][0][h];
#pragma unroll
                for (int r = 1; r < 8; r++) y[h] = add2(y[h], sums.v[t][r][h], one);
            }
            store_pair(p, rt.j, rt.row0, rt.live, first, count, n0 + t * 8 + 2 * q4, g4, unpack2(y[0]), unpack2(y[1]));
        }
    }
}

// grid (row_tiles-sized pieces of all jobs, groups or runs of tokens). Shared memory: the CTA's blocks as they are in memory
// | four warps' rings of activation fragments, SLOTS x 512 bytes each | activation scales [nb][8 MAXT].
template <int MAXT, int SLOTS, int MINB, bool FOLDED>
__global__ void __launch_bounds__(128, MINB) q6k_gemm_kernel(const GemmParams p) {
    static_assert(SLOTS / MAXT >= 2, "a block is read while the next is on its way");
    static_assert(SLOTS * 2048 >= 7 * 256 * 4, "the residues' sums of two tiles fit where the activations were");
    extern __shared__ __align__(16) uint8_t smem[];
    const int nb = p.nb, tid = threadIdx.x;
    const int j = job_of_tile(p, blockIdx.x);
    const int row_a = ((int)blockIdx.x - p.tile_begin[j]) * kGemmRows * p.row_tiles, live = min(p.row_tiles * kGemmRows, p.rows[j] - row_a);
    pdl_trigger();
    int first = 0, tile_lo = 0, count = p.n_tokens, tile_hi;
    size_t unit0 = (size_t)row_a * nb;
    if (p.gstart) {  // (groups never come folded; without the branch the folded form came out slower: a draft of 9 7504 / 7543 us)
        pdl_wait();
        prefetch_ahead<FOLDED>(p, p.prefetch_ahead);
        first = p.gstart[blockIdx.y];
        count = p.gcount[blockIdx.y];
        if (count <= 0) return;
        unit0 += (size_t)blockIdx.y * (size_t)p.expert_units;
        tile_hi = (count + 7) >> 3;
    } else {
        tile_lo = (int)blockIdx.y * p.run_tiles;
        tile_hi = min((count + 7) >> 3, tile_lo + p.run_tiles);
    }
    const size_t t_lo = unit0 >> 5, t_hi = (unit0 + (size_t)live * nb - 1) >> 5;
    const uint32_t s_raw = (uint32_t)__cvta_generic_to_shared(smem);
    {
        const uint8_t *src = p.w[j] + t_lo * kTileBytes;
        int n16 = (int)(t_hi - t_lo + 1) * (kTileBytes / 16);
        if (FOLDED) {
            const int tiles_j = (p.rows[j] + kGemmRows - 1) / kGemmRows;
            src = p.folded[j] + ((p.gstart ? (size_t)blockIdx.y * tiles_j : 0) + (size_t)(row_a / kGemmRows)) * (size_t)p.fold_tile_bytes;
            n16 = (int)(p.fold_tile_bytes >> 4);
        }
        for (int i = tid; i < n16; i += 128) copy_async16(s_raw + 16u * (uint32_t)i, src + 16 * (size_t)i);
        copy_commit();
    }
    if (!p.gstart) pdl_wait();
    float *s_ring = reinterpret_cast<float *>(smem + p.raw_bytes), *s_ad = s_ring + SLOTS * 512;
    for (int r0 = 0; r0 < live; r0 += kGemmRows) {
        const RowTile rt = {j, row_a + r0, min(kGemmRows, live - r0), s_raw, (int)(unit0 - (t_lo << 5)) + r0 * nb};
        const int tiles = tile_hi - tile_lo, groups = (tiles + MAXT - 1) / MAXT;
        for (int g = 0, t = tile_lo; g < groups; g++) {  // as few equal groups as MAXT allows
            const int nt = (tile_hi - t + groups - g - 1) / (groups - g);
#define LLAMD_TEAM(N)                                                                                                               \
    if constexpr (N <= MAXT) {                                                                                                      \
        if (nt == N) team_tiles<N, SLOTS, FOLDED>(p, rt, first, count, t, s_raw + (uint32_t)p.raw_bytes, s_ring, s_ad, 8 * MAXT, tid);       \
    }
            LLAMD_TEAM(1) LLAMD_TEAM(2) LLAMD_TEAM(3) LLAMD_TEAM(4) LLAMD_TEAM(5) LLAMD_TEAM(6) LLAMD_TEAM(7) LLAMD_TEAM(8)
#undef LLAMD_TEAM
            t += nt;
        }
    }
}

// grid as q6k_gemm_kernel's; a warp per BW blocks of a row tile, or (DIRECT) a warp per row tile, four row tiles a CTA.
// Shared memory: the blocks | the warps' activations, NT x BW x 2 KB each | the sums on their way from warp to warp (not DIRECT).
// (DIRECT at three blocks a row: 64896 bytes, three CTAs to an SM, where the launch bound of five costs 84 bytes of spills; two token
// tiles 89472 bytes, two CTAs.)
template <int NT, int BW, bool DIRECT, int THREADS, int MINB>
__global__ void __launch_bounds__(THREADS, MINB) q6k_gemm_few_kernel(const GemmParams p) {
    static_assert(DIRECT || NT == 1, "the sums that go from warp to warp are of one tile");
    extern __shared__ __align__(16) uint8_t smem[];
    const int nb = p.nb, tid = threadIdx.x, w = tid >> 5, lane = tid & 31, nw = blockDim.x >> 5;
    const int j = job_of_tile(p, blockIdx.x);
    const int row_a = ((int)blockIdx.x - p.tile_begin[j]) * kGemmRows * p.row_tiles, live = min(p.row_tiles * kGemmRows, p.rows[j] - row_a);
    int first = 0, tile_lo = 0, count = p.n_tokens, tile_hi;
    size_t unit0 = (size_t)row_a * nb;
    pdl_trigger();
    if (DIRECT && p.gstart) {
        pdl_wait();
        prefetch_ahead(p, p.prefetch_ahead);
        first = p.gstart[blockIdx.y];
        count = p.gcount[blockIdx.y];
        if (count <= 0) return;
        unit0 += (size_t)blockIdx.y * (size_t)p.expert_units;
        tile_hi = (count + 7) >> 3;
    } else {
        tile_lo = (int)blockIdx.y * p.run_tiles;
        tile_hi = min((count + 7) >> 3, tile_lo + p.run_tiles);
    }
    const size_t t_lo = unit0 >> 5, t_hi = (unit0 + (size_t)live * nb - 1) >> 5;
    const uint32_t s_raw = (uint32_t)__cvta_generic_to_shared(smem);
    {
        const uint8_t *src = p.w[j] + t_lo * kTileBytes;
        const int n16 = (int)(t_hi - t_lo + 1) * (kTileBytes / 16);
        for (int i = tid; i < n16; i += blockDim.x) copy_async16(s_raw + 16u * (uint32_t)i, src + 16 * (size_t)i);
        copy_commit();
    }
    if (!DIRECT || !p.gstart) pdl_wait();
    const uint32_t s_act = s_raw + (uint32_t)p.raw_bytes + (uint32_t)(w * NT * BW * 2048);
    float *s_x = reinterpret_cast<float *>(smem + p.raw_bytes + nw * NT * BW * 2048);
    const int r0 = DIRECT ? min(w * kGemmRows, ((live - 1) / kGemmRows) * kGemmRows) : 0;  // (a warp without a row tile repeats the last one)
    const RowTile rt = {j, row_a + r0, min(kGemmRows, live - r0), s_raw, (int)(unit0 - (t_lo << 5)) + r0 * nb};
    if constexpr (DIRECT) {
        for (int t = tile_lo; t < tile_hi; t += NT) {
            if (NT == 1 || tile_hi - t > 1) few_tiles<NT, BW, DIRECT>(p, rt, first, count, t, s_act, s_x, 0, nw, lane);
            else few_tiles<1, BW, DIRECT>(p, rt, first, count, t, s_act, s_x, 0, nw, lane);
        }
    } else {
        few_tiles<NT, BW, DIRECT>(p, rt, first, count, 0, s_act, s_x, w, nw, lane);
    }
}

// ---- short rows, many tokens per group ----
// With four blocks a row and less, a token group's preparation in q6k_gemm_kernel is as long as its products (down of 2048 tokens
// 519 us, here 471; 768: 236 / 226; 512: 164 / 180; of one and two blocks, 512 tokens: 104 / 99 and 148 / 131). Here a CTA folds its 16 rows
// into shared memory once, in operand order, and each of its warps takes token tiles of its own, all residues of them. FOLDED: it
// copies the rows' image.
constexpr int kTokStride = 80;  // words per staged token: 16-byte aligned, fragment reads in 32 banks
// CTAs to an SM: five, or where folding takes three blocks and more a row four with the registers it wants: down of 1024 / 2048 tokens 284
// 481 / 281 471, four blocks (1024 rows) 195 331 / 189 318; one block (2048 rows) 142 228 / 156 244.
template <bool FOLDED, int MINB>
__global__ void __launch_bounds__(128, MINB) q6k_gemm_shared_kernel(const GemmParams p) {
    extern __shared__ __align__(16) uint8_t smem[];
    const int nb = p.nb, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g4 = lane >> 2, q4 = lane & 3;
    uint4 *s_frag = reinterpret_cast<uint4 *>(smem);  // [block][residue][hi, lo][lane], or the image (kImageBlockBytes)
    float *s_d = reinterpret_cast<float *>(smem + (size_t)nb * 8 * 2 * 32 * 16);
    uint32_t *s_b = reinterpret_cast<uint32_t *>(s_d + kGemmRows * nb) + warp * 8 * kTokStride;
    const int j = job_of_tile(p, blockIdx.x), row0 = ((int)blockIdx.x - p.tile_begin[j]) * kGemmRows, rows = p.rows[j];
    pdl_trigger();
    pdl_wait();
    prefetch_ahead<FOLDED>(p, p.prefetch_ahead);
    const int first = p.gstart[blockIdx.y], count = p.gcount[blockIdx.y], live = min(kGemmRows, rows - row0);
    if (count <= 0) return;
    const size_t unit0 = (size_t)blockIdx.y * (size_t)p.expert_units + (size_t)row0 * nb;
    if (FOLDED) {
        const uint8_t *src = p.folded[j] + ((size_t)blockIdx.y * ((rows + kGemmRows - 1) / kGemmRows) + row0 / kGemmRows) * (size_t)p.fold_tile_bytes;
        const uint32_t dst = (uint32_t)__cvta_generic_to_shared(smem);
        for (int i = tid; i < (int)(p.fold_tile_bytes >> 4); i += 128) copy_async16(dst + 16u * (uint32_t)i, src + 16 * (size_t)i);
        copy_commit();
        copy_wait<0>();
    }
    for (int it = FOLDED ? 2 * kGemmRows * nb : tid; it < 2 * kGemmRows * nb; it += 128) {  // a thread: half of a (row, block)
        const int half = it >= kGemmRows * nb ? 1 : 0, rb = it - half * kGemmRows * nb, row = rb / nb, b = rb - row * nb;
        const size_t unit = unit0 + (size_t)min(row, live - 1) * nb + b;
        const uint8_t *tile = p.w[j] + (unit >> 5) * kTileBytes;
        const uint4 *cp = reinterpret_cast<const uint4 *>(tile) + t32_slot((int)(unit & 31));
        uint32_t S[24];
#pragma unroll
        for (int c = 0; c < 6; c++) {
            const uint4 v = __ldg(cp + (6 * half + c) * 32);
            S[4 * c] = v.x, S[4 * c + 1] = v.y, S[4 * c + 2] = v.z, S[4 * c + 3] = v.w;
        }
        const uint4 sc = __ldg(cp + kTileScaleOff / 16);
        if (half == 0) s_d[rb] = f16_bits_to_f32(__ldg(reinterpret_cast<const uint16_t *>(tile + kTileDOff) + (unit & 31)));
        const uint32_t scw[4] = {sc.x, sc.y, sc.z, sc.w};
#pragma unroll
        for (int q = 0; q < 4; q++) {
            Fold f;
            fold_scales(f, scw[q]);
#pragma unroll
            for (int k = 0; k < 2; k++) {
                const int quad = 4 * k + q;
                const uint32_t words[3] = {S[3 * quad], S[3 * quad + 1], S[3 * quad + 2]};
                uint32_t hi[2][4], lo[2][4];
                fold_quad(words, f, 0, hi, lo);
                // Lane L's 16 bytes sit in slot L ^ (L >> 3) ^ (b & 7): the threads of a warp here write the same word of
                // neighbouring rows and blocks, and the swizzle spreads them over all eight 16-byte bank groups.
                const int L = (row & 7) * 4 + q, P = L ^ (L >> 3) ^ (b & 7);
#pragma unroll
                for (int rr = 0; rr < 2; rr++) {
                    uint32_t *at = reinterpret_cast<uint32_t *>(s_frag + (size_t)((b * 8 + 4 * half + 2 * k + rr) * 2) * 32 + P) + (row >> 3);
                    at[0] = hi[rr][0], at[2] = hi[rr][2];
                    at[128] = lo[rr][0], at[130] = lo[rr][2];
                }
            }
        }
    }
    __syncthreads();
    const f32x2 one = p.one;
    const Quad zero = {{0, 0, 0, 0}};
    for (int n0 = warp * 8; n0 < count; n0 += 32) {
        auto act = [&](int tok) -> size_t {
            const int pt = first + min(n0 + tok, count - 1);
            return p.act_map ? (size_t)p.act_map[pt] : (size_t)pt;
        };
        const float *ad0 = p.ad + act(2 * q4) * nb, *ad1 = p.ad + act(2 * q4 + 1) * nb;
        const uint4 *src[4];  // staging: 8 tokens x 16 pieces of 16 bytes, four per lane
#pragma unroll
        for (int i = 0; i < 4; i++) src[i] = reinterpret_cast<const uint4 *>(p.aq_rm) + act((lane >> 4) + 2 * i) * nb * 16 + (lane & 15);
        uint32_t *put = s_b + (lane >> 4) * kTokStride + (lane & 15) * 4;
        f32x2 sum[8][2];
#pragma unroll
        for (int r = 0; r < 8; r++) sum[r][0] = sum[r][1] = 0ull;
        uint4 st[4];  // the next block's bytes wait in registers
#pragma unroll
        for (int i = 0; i < 4; i++) st[i] = __ldg(src[i]);
        f32x2 a = pack2(__ldg(ad0), __ldg(ad1));
        for (int b = 0; b < nb; b++) {
#pragma unroll
            for (int i = 0; i < 4; i++) *reinterpret_cast<uint4 *>(put + 2 * i * kTokStride) = st[i];
            __syncwarp();
            const float d0 = s_d[g4 * nb + b], d1 = s_d[(g4 + 8) * nb + b];
            const f32x2 dsc[2] = {mul2(pack2(d0, d0), a), mul2(pack2(d1, d1), a)};
            if (b + 1 < nb) {
#pragma unroll
                for (int i = 0; i < 4; i++) st[i] = __ldg(src[i] + (size_t)(b + 1) * 16);
                a = pack2(__ldg(ad0 + b + 1), __ldg(ad1 + b + 1));
            }
            const uint4 *fr = s_frag + (size_t)b * 8 * 2 * 32 + (FOLDED ? lane : lane ^ (lane >> 3) ^ (b & 7));
#pragma unroll
            for (int rp = 0; rp < 4; rp++) {
                const uint4 bw = *reinterpret_cast<const uint4 *>(s_b + g4 * kTokStride + rp * 16 + q4 * 4);
#pragma unroll
                for (int rr = 0; rr < 2; rr++) {
                    const int at = FOLDED ? 4 * rp + rr : 2 * (2 * rp + rr);
                    const uint4 h4 = fr[at * 32], l4 = fr[(at + (FOLDED ? 2 : 1)) * 32];
                    const uint32_t ah[4] = {h4.x, h4.y, h4.z, h4.w}, al[4] = {l4.x, l4.y, l4.z, l4.w};
                    int ch[4], cl[4];
                    mma_8<false>(ch, ah, rr ? bw.z : bw.x, rr ? bw.w : bw.y, zero);
                    mma_8<true>(cl, al, rr ? bw.z : bw.x, rr ? bw.w : bw.y, zero);
#pragma unroll
                    for (int h = 0; h < 2; h++) {  // (|aux| < 2^24: exact as a float)
                        const f32x2 aux = pack2((float)(ch[2 * h] * 64 + (cl[2 * h] >> 2)), (float)(ch[2 * h + 1] * 64 + (cl[2 * h + 1] >> 2)));
                        sum[2 * rp + rr][h] = add2(sum[2 * rp + rr][h], mul2(dsc[h], aux), one);
                    }
                }
            }
            __syncwarp();
        }
        f32x2 y[2];
#pragma unroll
        for (int h = 0; h < 2; h++) {
            y[h] = sum[0][h];
#pragma unroll
            for (int r = 1; r < 8; r++) y[h] = add2(y[h], sum[r][h], one);
        }
        store_pair(p, j, row0, live, first, count, n0 + 2 * q4, g4, unpack2(y[0]), unpack2(y[1]));
    }
}

// Folds every (expert, row tile) of one matrix once and keeps the image: grid (row tiles, experts), a warp per residue pair.
__global__ void __launch_bounds__(128) q6k_prefold_kernel(const uint8_t *__restrict__ w, uint8_t *__restrict__ dst, int rows, int nb,
                                                          long long expert_units, long long tile_bytes) {
    extern __shared__ __align__(16) uint8_t smem[];
    const int tid = threadIdx.x, rp = tid >> 5, lane = tid & 31, g4 = lane >> 2, q4 = lane & 3, row0 = blockIdx.x * kGemmRows;
    const int live = min(kGemmRows, rows - row0);
    const size_t unit0 = (size_t)blockIdx.y * (size_t)expert_units + (size_t)row0 * nb;
    const size_t t_lo = unit0 >> 5, t_hi = (unit0 + (size_t)live * nb - 1) >> 5;
    const uint32_t s_raw = (uint32_t)__cvta_generic_to_shared(smem);
    const int n16 = (int)(t_hi - t_lo + 1) * (kTileBytes / 16);
    for (int i = tid; i < n16; i += 128) copy_async16(s_raw + 16u * (uint32_t)i, w + t_lo * kTileBytes + 16 * (size_t)i);
    copy_commit();
    copy_wait<0>();
    __syncthreads();
    uint8_t *out = dst + ((size_t)blockIdx.y * gridDim.x + blockIdx.x) * (size_t)tile_bytes;
    uint32_t word_off[3];
    fold_offsets(rp, q4, word_off);
    for (int b = 0; b < nb; b++) {
        uint32_t hi[2][4], lo[2][4];
#pragma unroll
        for (int h = 0; h < 2; h++) {
            float d;
            const int m = g4 + 8 * h;
            fold_block(s_raw, (int)(unit0 - (t_lo << 5)) + min(m, live - 1) * nb + b, q4, word_off, h, hi, lo, d);
            if (rp == 0 && q4 == 0) reinterpret_cast<float *>(out + (size_t)nb * kImageBlockBytes)[m * nb + b] = m < live ? d : 0.0f;
        }
        uint4 *o = reinterpret_cast<uint4 *>(out + (size_t)b * kImageBlockBytes + rp * 2048) + lane;
#pragma unroll
        for (int rr = 0; rr < 2; rr++) {
            o[rr * 32] = make_uint4(hi[rr][0], hi[rr][1], hi[rr][2], hi[rr][3]);
            o[64 + rr * 32] = make_uint4(lo[rr][0], lo[rr][1], lo[rr][2], lo[rr][3]);
        }
    }
}

}  // namespace llamd

using namespace llamd;

// KERNEL: one launch configuration remembers its own limits
template <auto KERNEL>
static void gemm_launch_k(GemmParams &p, int n_groups, int threads, size_t smem) {
    static size_t configured = 0;
    if (smem > 48 * 1024 && smem > configured) {
        const cudaError_t e = cudaFuncSetAttribute(KERNEL, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) {
            cudaGetLastError();  // (a refusal of this launch, not of the next one)
            set_error(e, "q6k gemm: shared memory attribute");
            return;
        }
        configured = smem;
    }
    int grid_x = 0;
    for (int i = 0; i < p.njobs; i++) {
        p.tile_begin[i] = grid_x;
        grid_x += (p.rows[i] + kGemmRows * p.row_tiles - 1) / (kGemmRows * p.row_tiles);
    }
    if (p.gstart) {
        static size_t cached_smem = 0;
        static int cached_slots = 0;
        if (cached_smem != smem) {
            int dev = 0, sms = 0, per_sm = 0;
            cudaGetDevice(&dev);
            cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, KERNEL, threads, smem);
            cached_slots = sms * (per_sm > 0 ? per_sm : 1);
            cached_smem = smem;
        }
        p.prefetch_ahead = cached_slots;
    }
    launch_kc(p.gstart ? PDL_OTHER : PDL_MATVEC, "q6k_gemm", KERNEL, dim3(grid_x, n_groups), dim3(threads), smem, p);
}
constexpr size_t kMaxSmem = 227 * 1024;  // what a CTA may have
template <int MAXT, int SLOTS>
static size_t team_smem(const GemmParams &p) {
    return (size_t)p.raw_bytes + (size_t)SLOTS * 2048 + (size_t)p.nb * 8 * MAXT * 4;
}
template <int MAXT, int SLOTS, int MINB, bool FOLDED>
static void gemm_launch_t(GemmParams &p, int n_groups) {
    gemm_launch_k<q6k_gemm_kernel<MAXT, SLOTS, MINB, FOLDED>>(p, n_groups, 128, team_smem<MAXT, SLOTS>(p));
}
template <int NT, int BW, bool DIRECT, int THREADS, int MINB>
static void gemm_launch_few(GemmParams &p, int n_groups) {
    const int warps = DIRECT ? p.row_tiles : (p.nb + BW - 1) / BW;
    gemm_launch_k<q6k_gemm_few_kernel<NT, BW, DIRECT, THREADS, MINB>>(p, n_groups, 32 * warps, (size_t)p.raw_bytes + (size_t)warps * NT * BW * 2048 + (DIRECT ? 0 : 4096));
}

template <bool FOLDED, int MINB>
static void shared_launch(GemmParams &p, int n_groups) {
    p.row_tiles = 1;
    gemm_launch_k<q6k_gemm_shared_kernel<FOLDED, MINB>>(p, n_groups, 128, (size_t)p.nb * 8 * 2 * 32 * 16 + (size_t)kGemmRows * p.nb * 4 + 4 * 8 * kTokStride * 4);
}

// Shared memory for `units` consecutive blocks: whole tiles, one more where they need not start with one.
static int raw_tile_bytes(int units, bool aligned) {
    return (aligned && units % 32 == 0 ? units / 32 : (units + 30) / 32 + 1) * kTileBytes;
}

// n_groups > 0: that many token groups of about `tokens` each. 0: one group of p.n_tokens.
static void gemm_launch(GemmParams &p, int n_groups, int tokens) {
    // Groups take the images of short rows, for as many tokens as a warp per token tile pays for: folding on the way is faster
    // everywhere else. us, stored blocks / images, by blocks a row and tokens per group: 1 (2048 rows) 12 tokens 38 / 68, 32: 99 / 89,
    // 128: 227 / 211; 3 (2048) 12: 95 / 130, 32: 169 / 162, 128: 472 / 433; 4 (1024) 12: 71 / 87, 32: 114 / 107, 128: 318 / 290; 5 (1024)
    // 32: 131 / 136, 44: 161 / 173, 64: 222 / 213, 128: 397 / 366; 6 (1024) 64: 243 / 277, 128: 439 / 471; 8 (2 x 768) 32: 257 / 318, 128: 806 / 878.
    const bool images = p.gstart && p.folded[0] && p.nb <= kPrefoldBlocks && tokens > (p.nb < 5 ? 24 : 48);
    const bool folded = !p.gstart && p.folded[0];
    if (p.nb < 1 || p.nb > (n_groups ? kGroupedBlocks : folded ? kFoldedBlocks : kGemmBlocks)) {
        set_error_msg(n_groups ? "q6k gemm: blocks per row must be 1..26" : folded ? "q6k gemm: blocks per folded row must be 1..25"
                                                                                    : "q6k gemm: blocks per row must be 1..24");
        return;
    }
    if (n_groups > 65535) {
        set_error_msg("q6k gemm: too many groups");
        return;
    }
    p.one = kOne2;
    const int tiles = (tokens + 7) / 8;
    const bool direct = !folded && p.nb <= 3 && tokens <= 16, few = direct || (!folded && !p.gstart && tiles <= 1);
    p.row_tiles = direct ? 4 : folded || few || p.nb >= 6 ? 1 : (p.nb >= 3 ? 2 : 4);
    p.fold_tile_bytes = (long long)expert_fold_tile_bytes(p.nb);
    p.raw_bytes = folded ? (int)p.fold_tile_bytes : raw_tile_bytes(p.row_tiles * kGemmRows * p.nb, !n_groups || p.expert_units % 32 == 0);
    if (!n_groups) {
        p.run_tiles = tiles <= 8 ? tiles : 8;
        n_groups = (tiles + p.run_tiles - 1) / p.run_tiles;
        if (n_groups > 65535) {
            set_error_msg("q6k gemm: too many tokens");
            return;
        }
    }
    // The lines lie where the forms' times cross, see there; MAXT and the CTAs per SM by us of gate and up: 64 tokens (half a tile per
    // expert) <2, 4, 6> 124, <4, 8, 5> 136; 512 (four) <8, 16, 3> 257, <6, 12, 4> 267, <4, 8, 4> 285; down of 512 <6, 12, 4> 164, <8, 16, 3> 179.
    if (folded) {
        // (an image of 24 blocks a row leaves no room for the rings of eight tiles)
        if (tiles <= 4 || team_smem<8, 16>(p) > kMaxSmem) gemm_launch_t<4, 8, 2, true>(p, n_groups);
        else gemm_launch_t<8, 16, 2, true>(p, n_groups);
    } else if (images) {
        shared_launch<true, 5>(p, n_groups);
    } else if (direct) {
        if (tiles <= 1) gemm_launch_few<1, 3, true, 128, 5>(p, n_groups);
        else gemm_launch_few<2, 3, true, 128, 3>(p, n_groups);
    } else if (few) {
        if (p.nb <= 8) gemm_launch_few<1, 2, false, 128, 4>(p, n_groups);
        else if (p.nb <= 16) gemm_launch_few<1, 2, false, 256, 2>(p, n_groups);
        else gemm_launch_few<1, 2, false, 384, 1>(p, n_groups);
    } else if (p.gstart && p.nb <= 2 && tokens > 24) {
        shared_launch<false, 5>(p, n_groups);
    } else if (p.gstart && p.nb <= 4 && tokens > 40) {
        shared_launch<false, 4>(p, n_groups);
    } else if (tiles <= 1) {
        gemm_launch_t<2, 4, 6, false>(p, n_groups);
    } else if (tiles <= 3) {
        gemm_launch_t<4, 8, 4, false>(p, n_groups);
    } else if (p.nb <= 4) {
        gemm_launch_t<6, 12, 4, false>(p, n_groups);
    } else {
        gemm_launch_t<8, 16, 3, false>(p, n_groups);
    }
}

extern "C" {

// Q8_K quants [nblocks][256] (natural order) -> the operand-order words the GEMM reads.
void llamd_fwd_q8k_residue_major(const int8_t *aq, void *aq_rm, size_t nblocks) {
    if (!nblocks) return;
    const size_t n = nblocks * 64;
    launch_k("q8k_residue_major", q8k_residue_major_kernel, dim3((unsigned)((n + 255) / 256)), dim3(256), 0, aq, (uint32_t *)aq_rm, nblocks);
}

// Up to three matrices (w1/w2 may be NULL) against ntok activations; outputs [ntok][rows_i].
// Same results as llamd_fwd_matvec_tokens, on the integer tensor path.
void llamd_fwd_gemm_tokens(const void *w0, const void *w1, const void *w2, const void *aq_rm, const float *ad, float *o0, float *o1,
                           float *o2, int blocks, int rows0, int rows1, int rows2, int ntok) {
    if (ntok < 1) return;
    GemmParams p = {};
    p.w[0] = (const uint8_t *)w0; p.w[1] = (const uint8_t *)w1; p.w[2] = (const uint8_t *)w2;
    p.out[0] = o0; p.out[1] = o1; p.out[2] = o2;
    p.rows[0] = rows0; p.rows[1] = rows1; p.rows[2] = rows2;
    p.njobs = w2 ? 3 : (w1 ? 2 : 1);
    p.nb = blocks;
    p.aq_rm = (const uint32_t *)aq_rm;
    p.ad = ad;
    p.n_tokens = ntok;
    gemm_launch(p, 0, ntok);
}

// Expert-major grouped GEMM over the scatter plan (gstart/gcount per expert, pairs sorted by expert):
// pair p reads activation act_map[p] and writes out[pslot[p]][rows]. wb/ob may be NULL.
// Same results as llamd_fwd_expert_major.
void llamd_fwd_expert_gemm(const void *wa, const void *wb, const int32_t *gstart, const int32_t *gcount, const int32_t *act_map,
                           const int32_t *pslot, const void *aq_rm, const float *ad, float *oa, float *ob, int blocks, int rows,
                           int n_expert) {
    expert_gemm_scatter(wa, wb, gstart, gcount, act_map, pslot, aq_rm, ad, oa, ob, blocks, rows, n_expert, 0, nullptr, 1);
}

}  // extern "C"

size_t llamd::expert_fold_tile_bytes(int blocks) { return (size_t)blocks * kImageBlockBytes + (size_t)kGemmRows * blocks * 4; }
size_t llamd::expert_fold_bytes(int blocks, int rows, int n_expert) {
    return expert_fold_tile_bytes(blocks) * (size_t)((rows + kGemmRows - 1) / kGemmRows) * (size_t)n_expert;
}
void llamd::expert_prefold(const void *w, void *dst, int blocks, int rows, int n_expert) {
    if (n_expert > 65535 || n_expert < 1 || rows < 1 || blocks < 1 || blocks > kFoldedBlocks) {
        set_error_msg("expert prefold: 1..65535 experts, rows positive, 1..25 blocks per row");
        return;
    }
    const size_t smem = (size_t)raw_tile_bytes(kGemmRows * blocks, false);
    static size_t configured = 0;
    if (smem > 48 * 1024 && smem > configured) {
        if (cudaFuncSetAttribute(q6k_prefold_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) {
            set_error_msg("expert prefold: shared memory attribute");
            return;
        }
        configured = smem;
    }
    launch_k("q6k_prefold", q6k_prefold_kernel, dim3((rows + kGemmRows - 1) / kGemmRows, n_expert), dim3(128), smem, (const uint8_t *)w,
             (uint8_t *)dst, rows, blocks, (long long)rows * blocks, (long long)expert_fold_tile_bytes(blocks));
}

void llamd::expert_gemm_scatter(const void *wa, const void *wb, const int32_t *gstart, const int32_t *gcount, const int32_t *act_map,
                                const int32_t *pslot, const void *aq_rm, const float *ad, float *oa, float *ob, int blocks, int rows,
                                int n_expert, int pairs, float *const *out_tab, int out_div, const void *fa, const void *fb) {
    if (out_tab && (wb || out_div < 1)) {
        set_error_msg("expert gemm: scattered outputs take one matrix and a positive row-block count per GPU");
        return;
    }
    if (n_expert < 1) return;
    GemmParams p = {};
    p.out_tab = out_tab;
    p.out_div = out_div;
    p.w[0] = (const uint8_t *)wa; p.w[1] = (const uint8_t *)wb;
    p.folded[0] = (const uint8_t *)fa; p.folded[1] = wb ? (const uint8_t *)fb : nullptr;
    p.out[0] = oa; p.out[1] = ob;
    p.rows[0] = rows; p.rows[1] = rows;
    p.njobs = wb ? 2 : 1;
    p.nb = blocks;
    p.aq_rm = (const uint32_t *)aq_rm;
    p.ad = ad;
    p.gstart = gstart; p.gcount = gcount; p.act_map = act_map; p.out_map = pslot;
    p.expert_units = (long long)rows * blocks;
    gemm_launch(p, n_expert, pairs > 0 ? (pairs + n_expert - 1) / n_expert : 64);
}

// Up to three matrices kept folded (expert_prefold with one "expert" each) against ntok activations: out_i[ntok][rows_i].
// 2 bytes per weight and no folding. Same results as llamd_fwd_gemm_tokens.
void llamd::gemm_tokens_folded3(const void *f0, const void *f1, const void *f2, const void *aq_rm, const float *ad, float *o0, float *o1,
                                float *o2, int blocks, int rows0, int rows1, int rows2, int ntok) {
    if (ntok < 1) return;
    GemmParams p = {};
    p.folded[0] = (const uint8_t *)f0; p.folded[1] = (const uint8_t *)f1; p.folded[2] = (const uint8_t *)f2;
    p.out[0] = o0; p.out[1] = o1; p.out[2] = o2;
    p.rows[0] = rows0; p.rows[1] = rows1; p.rows[2] = rows2;
    p.njobs = f2 ? 3 : (f1 ? 2 : 1);
    p.nb = blocks;
    p.aq_rm = (const uint32_t *)aq_rm;
    p.ad = ad;
    p.n_tokens = ntok;
    gemm_launch(p, 0, ntok);
}
void llamd::gemm_tokens_folded(const void *folded, const void *aq_rm, const float *ad, float *out, int blocks, int rows, int ntok) {
    gemm_tokens_folded3(folded, nullptr, nullptr, aq_rm, ad, out, nullptr, nullptr, blocks, rows, 0, 0, ntok);
}
