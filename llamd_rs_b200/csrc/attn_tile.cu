// Attention for the tokens of one prefill tile, as three register-tiled kernels.
//
// The arithmetic is that of `attend` (crates/llamd-cpu/src/lib.rs, the per-head
// loop: dot = sum_d q[d]*k[t][d] from 0.0 in d order, logit = dot*scale,
// softmax with an ordered sum, out[d] = sum_t (e[t]*inv)*v[t][d] from 0.0 in t
// order), one query per token, every token seeing positions 0..pos of the ONE
// cache the tile has already stored into. Nothing is re-associated: each
// output element is one thread-private accumulator that walks its reduction
// index in order with an unfused multiply and add. What changes against the
// per-token kernels is only WHO holds the chains: a thread owns a 4x4 (scores)
// or 4x8 (output) patch of independent chains, so operands fetched from shared
// memory are reused 4-8 times and the FP32 pipe, not memory, sets the pace.
//
//   tile_scores_kernel   S[t][p] = scale * (q_t . k_p)        64 tokens x 64 positions x one head per CTA
//   tile_softmax_kernel  W[t][p] = exp(S - max) / sum          one warp per (token, head) row, in place
//   tile_pv_kernel       out[t][d] = sum_p W[t][p] * v_p[d]    32 tokens x head_dim x one head per CTA
//
// A weight beyond a token's own position is staged as +0.0, and 0*v added to
// an accumulator that started at +0.0 leaves it unchanged, so every token's
// chain is exactly the chain over its own positions.
#include "common.cuh"
#include "packed_f32.cuh"
#include "quant.cuh"

namespace llamd {
namespace {

__device__ __forceinline__ void cp_async16(void *dst, const void *src, int bytes) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Two chains per instruction (packed_f32.cuh). The FP32 pipe does as many operations a cycle either way, but at two a scalar
// instruction left no issue slots for the shared-memory loads: us a 512-token piece of a 2000-token prompt, scalar / packed:
// scores 199 / 181, values 214 / 200.
__device__ __forceinline__ f32x2 mul_add2(f32x2 a, f32x2 b, f32x2 s, f32x2 one) { return add2(s, mul2(a, b), one); }  // s + a*b, each rounded

constexpr int kST = 64;  // tokens per CTA of the score kernel
constexpr int kSP = 64;  // positions per CTA of the score kernel

// grid (position tiles, token tiles, heads), 256 threads.
// Thread (ty, tx) = (tid / 16, tid % 16) owns tokens 4ty..4ty+3 and positions tx, tx+16, tx+32, tx+48 of the tile:
// two token pairs, whose queries lie interleaved in shared memory, against four keys.
__global__ void __launch_bounds__(256) tile_scores_kernel(const float *__restrict__ q, const float *__restrict__ kc, float *__restrict__ scores,
                                                          int n_head, int n_head_kv, int hd, const int32_t *__restrict__ meta, int max_kv,
                                                          int ntok, f32x2 one) {
    extern __shared__ __align__(16) float sm[];
    __shared__ int s_pos[kST];
    pdl_trigger();
    pdl_wait();
    const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
    const int p0 = blockIdx.x * kSP, t0 = blockIdx.y * kST, h = blockIdx.z;
    if (tid < kST) s_pos[tid] = (t0 + tid < ntok) ? meta[2 * (t0 + tid) + 1] : -1;
    __syncthreads();
    int maxpos = -1;
    for (int i = 0; i < kST; i++) maxpos = max(maxpos, s_pos[i]);
    if (p0 > maxpos) return;
    const int S = hd + 4;  // row stride: 16-byte aligned, rows 4 apart fall into different bank groups
    const int SQ = 2 * hd + 4;  // ... of a token pair: (even, odd) for every column
    float *sQ = sm, *sK = sm + (kST / 2) * SQ;
    const int hd4 = hd >> 2, kv_dim = n_head_kv * hd, kvh = h / (n_head / n_head_kv);
    for (int idx = tid; idx < kST * hd4; idx += 256) {
        const int r = idx / hd4, c = idx - r * hd4;
        const int p = p0 + r;
        cp_async16(sK + r * S + 4 * c, kc + (size_t)min(p, maxpos) * kv_dim + (size_t)kvh * hd + 4 * c, p <= maxpos ? 16 : 0);
    }
    cp_async_commit();
    for (int idx = tid; idx < (kST / 2) * hd4; idx += 256) {
        const int r = idx / hd4, c = idx - r * hd4, t = t0 + 2 * r;
        const float4 *q0 = reinterpret_cast<const float4 *>(q + ((size_t)min(t, ntok - 1) * n_head + h) * hd) + c;
        const float4 *q1 = reinterpret_cast<const float4 *>(q + ((size_t)min(t + 1, ntok - 1) * n_head + h) * hd) + c;
        const float4 a = *q0, b = *q1;  // (a token past the end scores like the last one; its rows are not stored)
        float4 *d = reinterpret_cast<float4 *>(sQ + r * SQ + 8 * c);
        d[0] = make_float4(a.x, b.x, a.y, b.y);
        d[1] = make_float4(a.z, b.z, a.w, b.w);
    }
    cp_async_wait<0>();
    __syncthreads();
    f32x2 acc[2][4];
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = 0ull;
    const float *qb = sQ + (ty * 2) * SQ, *kb = sK + tx * S;
#pragma unroll 2
    for (int d4 = 0; d4 < hd4; d4++) {
        ulonglong2 a[2][2];
        float4 b[4];
#pragma unroll
        for (int i = 0; i < 2; i++) {
            a[i][0] = *reinterpret_cast<const ulonglong2 *>(qb + i * SQ + 8 * d4);
            a[i][1] = *reinterpret_cast<const ulonglong2 *>(qb + i * SQ + 8 * d4 + 4);
        }
#pragma unroll
        for (int j = 0; j < 4; j++) b[j] = *reinterpret_cast<const float4 *>(kb + j * 16 * S + 4 * d4);
#pragma unroll
        for (int c = 0; c < 4; c++) {
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const float k = c == 0 ? b[j].x : c == 1 ? b[j].y : c == 2 ? b[j].z : b[j].w;
                const f32x2 kk = pack2(k, k);
#pragma unroll
                for (int i = 0; i < 2; i++) acc[i][j] = mul_add2(c & 1 ? a[i][c >> 1].y : a[i][c >> 1].x, kk, acc[i][j], one);
            }
        }
    }
    const float scale = __fdiv_rn(1.0f, __fsqrt_rn((float)hd));
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int t = t0 + ty * 4 + i, pos = s_pos[ty * 4 + i];
        float *row = scores + ((size_t)t * n_head + h) * max_kv;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int p = p0 + j * 16 + tx;
            const float2 v = unpack2(acc[i >> 1][j]);
            if (p <= pos) row[p] = __fmul_rn(i & 1 ? v.y : v.x, scale);
        }
    }
}

// One warp per (token, head) row: the logits become the softmax weights e*inv in place. The rows' sums are walked side by
// side by the first warp, a lane per row (a warp per chain is one lane's adds at a whole warp's issue; the kernel is bound by
// issue, most of it the exponentials): with a warp per chain a prompt of 1999 tokens took 0.5 % longer.
// Dynamic shared memory: [warps][n_cap] floats, n_cap = 4 mod 32 (the lanes' 16-byte reads meet different banks).
__global__ void tile_softmax_kernel(float *__restrict__ scores, const int32_t *__restrict__ meta, int n_head, int max_kv, int ntok, int n_cap) {
    extern __shared__ __align__(16) float sm[];
    __shared__ float s_inv[8];
    pdl_trigger();
    pdl_wait();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
    const int row = blockIdx.x * warps + warp, rows = ntok * n_head;
    const int n = row < rows ? min(meta[2 * (row / n_head) + 1] + 1, n_cap) : 0;
    float *sl = sm + (size_t)warp * n_cap;
    float *g = scores + (size_t)row * max_kv;
    float lmax = -INFINITY;
    for (int p = lane; p < n; p += 32) {
        const float l = g[p];
        sl[p] = l;
        lmax = fmaxf(lmax, l);
    }
    for (int off = 16; off > 0; off >>= 1) lmax = fmaxf(lmax, __shfl_xor_sync(0xffffffffu, lmax, off));
    for (int p = lane; p < n; p += 32) sl[p] = ref_expf(__fsub_rn(sl[p], lmax));
    __syncthreads();
    if (warp == 0 && lane < warps) {
        const int r = blockIdx.x * warps + lane;
        if (r < rows) s_inv[lane] = __fdiv_rn(1.0f, chain_sum(sm + (size_t)lane * n_cap, min(meta[2 * (r / n_head) + 1] + 1, n_cap), 0.0f));
    }
    __syncthreads();
    const float inv = s_inv[warp];
    for (int p = lane; p < n; p += 32) g[p] = __fmul_rn(sl[p], inv);
}

constexpr int kOT = 32;  // tokens per CTA of the output kernel
constexpr int kOP = 32;  // positions per staged tile
constexpr int kWS = kOP + 4;

// grid (token tiles, heads), 128 threads. Thread (ty, tx) = (tid / 16, tid % 16) owns tokens 4ty..4ty+3 and the
// output columns 64g + 4tx .. +3 for g < HD/64.
template <int HD>
__global__ void __launch_bounds__(128) tile_pv_kernel(const float *__restrict__ w, const float *__restrict__ vc, float *__restrict__ out, int n_head,
                                                      int n_head_kv, const int32_t *__restrict__ meta, int max_kv, int ntok, f32x2 one) {
    constexpr int G = HD / 64, HD4 = HD / 4;
    __shared__ __align__(16) float sW[2][kOT][kWS];
    __shared__ __align__(16) float sV[2][kOP][HD];
    __shared__ int s_pos[kOT];
    pdl_trigger();
    pdl_wait();
    const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
    const int t0 = ((int)gridDim.x - 1 - (int)blockIdx.x) * kOT, h = blockIdx.y;  // the longest tiles start first
    if (tid < kOT) s_pos[tid] = (t0 + tid < ntok) ? meta[2 * (t0 + tid) + 1] : -1;
    __syncthreads();
    int maxpos = -1;
    for (int i = 0; i < kOT; i++) maxpos = max(maxpos, s_pos[i]);
    const int kv_dim = n_head_kv * HD, kvh = h / (n_head / n_head_kv);
    const float *vb = vc + (size_t)kvh * HD;
    auto stage = [&](int pt, int buf) {
        for (int idx = tid; idx < kOT * (kOP / 4); idx += 128) {
            const int r = idx / (kOP / 4), c = idx - r * (kOP / 4);
            const int p = pt * kOP + 4 * c;
            const int valid = max(0, min(4, s_pos[r] - p + 1));
            const float *src = valid ? w + ((size_t)(t0 + r) * n_head + h) * max_kv + p : w;
            cp_async16(&sW[buf][r][4 * c], src, 4 * valid);
        }
        for (int idx = tid; idx < kOP * HD4; idx += 128) {
            const int r = idx / HD4, c = idx - r * HD4;
            const int p = pt * kOP + r;
            cp_async16(&sV[buf][r][4 * c], vb + (size_t)min(p, maxpos) * kv_dim + 4 * c, p <= maxpos ? 16 : 0);
        }
        cp_async_commit();
    };
    f32x2 acc[4][G * 2];
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int c = 0; c < G * 2; c++) acc[i][c] = 0ull;
    const int n_pt = maxpos / kOP + 1;  // maxpos >= 0: the tile holds at least one token
    stage(0, 0);
    for (int pt = 0; pt < n_pt; pt++) {
        const int buf = pt & 1;
        if (pt + 1 < n_pt) {
            stage(pt + 1, buf ^ 1);
            cp_async_wait<1>();
        } else {
            cp_async_wait<0>();
        }
        __syncthreads();
#pragma unroll 2
        for (int p4 = 0; p4 < kOP / 4; p4++) {
            float4 wv[4];
#pragma unroll
            for (int i = 0; i < 4; i++) wv[i] = *reinterpret_cast<const float4 *>(&sW[buf][ty * 4 + i][4 * p4]);
#pragma unroll
            for (int c = 0; c < 4; c++) {
                ulonglong2 v[G];
#pragma unroll
                for (int g = 0; g < G; g++) v[g] = *reinterpret_cast<const ulonglong2 *>(&sV[buf][4 * p4 + c][64 * g + 4 * tx]);
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const float wi = c == 0 ? wv[i].x : c == 1 ? wv[i].y : c == 2 ? wv[i].z : wv[i].w;
                    const f32x2 ww = pack2(wi, wi);
#pragma unroll
                    for (int g = 0; g < G; g++) {
                        acc[i][2 * g] = mul_add2(ww, v[g].x, acc[i][2 * g], one);
                        acc[i][2 * g + 1] = mul_add2(ww, v[g].y, acc[i][2 * g + 1], one);
                    }
                }
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int t = t0 + ty * 4 + i;
        if (t < ntok) {
#pragma unroll
            for (int g = 0; g < G; g++)
                *reinterpret_cast<ulonglong2 *>(out + ((size_t)t * n_head + h) * HD + 64 * g + 4 * tx) = make_ulonglong2(acc[i][2 * g], acc[i][2 * g + 1]);
        }
    }
}

}  // namespace
}  // namespace llamd

using namespace llamd;

extern "C" {
// The tiled form of llamd_fwd_attention_tile. n_kv_max bounds pos+1 over the tile's tokens (the host knows it:
// base position + token count); the kernels read each token's own position from meta[2i+1].
// Shapes the tiled kernels do not cover (head_dim other than 64 or 128, max_kv not a multiple of 4, a context
// beyond one row of shared memory) go to the per-token kernels, which compute the same bits.
void llamd_fwd_attention_prefill(const float *q, const float *kc, const float *vc, float *out, float *scores, int n_head, int n_head_kv,
                                 int hd, const int32_t *meta, int max_kv, int ntok, int n_kv_max) {
    if (ntok <= 0) return;
    const int n_cap = ((n_kv_max + 31) & ~31) + 4;
    const bool tiled = scores && (hd == 64 || hd == 128) && max_kv % 4 == 0 && n_kv_max > 0 && n_kv_max <= max_kv && n_head_kv > 0 &&
                       n_head % n_head_kv == 0 && (size_t)n_cap * 4 <= 200 * 1024;
    if (!tiled) {
        llamd_fwd_attention_tile(q, kc, vc, out, scores, n_head, n_head_kv, hd, meta, max_kv, ntok);
        return;
    }
    const size_t smem_s = (size_t)(kST / 2 * (2 * hd + 4) + kSP * (hd + 4)) * sizeof(float);
    static size_t conf_s = 0;
    if (smem_s > 48 * 1024 && smem_s > conf_s) {
        cudaFuncSetAttribute(tile_scores_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_s);
        conf_s = smem_s;
    }
    launch_k("tile_scores", tile_scores_kernel, dim3((n_kv_max + kSP - 1) / kSP, (ntok + kST - 1) / kST, n_head), dim3(256), smem_s, q, kc, scores,
             n_head, n_head_kv, hd, meta, max_kv, ntok, kOne2);
    int warps = (int)((200 * 1024) / ((size_t)n_cap * 4));
    warps = warps > 8 ? 8 : warps;
    const size_t smem_m = (size_t)warps * n_cap * sizeof(float);
    static size_t conf_m = 0;
    if (smem_m > 48 * 1024 && smem_m > conf_m) {
        cudaFuncSetAttribute(tile_softmax_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_m);
        conf_m = smem_m;
    }
    const int rows = ntok * n_head;
    launch_k("tile_softmax", tile_softmax_kernel, dim3((rows + warps - 1) / warps), dim3(32 * warps), smem_m, scores, meta, n_head, max_kv, ntok, n_cap);
    const dim3 grid((ntok + kOT - 1) / kOT, n_head);
    if (hd == 64)
        launch_k("tile_pv", tile_pv_kernel<64>, grid, dim3(128), 0, (const float *)scores, vc, out, n_head, n_head_kv, meta, max_kv, ntok, kOne2);
    else
        launch_k("tile_pv", tile_pv_kernel<128>, grid, dim3(128), 0, (const float *)scores, vc, out, n_head, n_head_kv, meta, max_kv, ntok, kOne2);
}
}
