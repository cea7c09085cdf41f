// Attention for the tokens of one prefill tile, as three register-tiled kernels.
//
// The arithmetic is that of `attend` (crates/llamd-cpu/src/lib.rs, the per-head
// loop: dot = sum_d q[d]*k[t][d] from 0.0 in d order, logit = dot*scale,
// softmax with an ordered sum, out[d] = sum_t (e[t]*inv)*v[t][d] from 0.0 in t
// order), one query per token, every token seeing positions 0..pos of the ONE
// cache the tile has already stored into. Nothing is re-associated: each
// output element is one thread-private accumulator that walks its reduction
// index in order with an unfused multiply and add. What changes against the
// per-token kernels is only WHO holds the chains: a thread owns an 8x4 (scores)
// or 4x4 (output) patch of independent chains, so operands fetched from shared
// memory are reused 4-8 times and the FP32 pipe, not memory, sets the pace.
//
//   tile_scores_kernel   S[t][p] = scale * (q_t . k_p)        64 tokens x 128 positions x one head per CTA
//   tile_softmax_kernel  W[t][p] = exp(S - max) / sum          one warp per (token, head) row, in place
//   tile_pv_kernel       out[t][d] = sum_p W[t][p] * v_p[d]    16 tokens x head_dim x one head per CTA
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

// Two chains per instruction (packed_f32.cuh). The FP32 pipe takes two cycles for a packed instruction, as for two scalar ones
// (2.1 to 2.5 measured, with the operands' registers); what packing saves is issue. Scalar multiplies feeding packed adds, which
// need no value twice, took as long for the scores and 4 % longer for the values; all scalar 6 and 10 % longer.
__device__ __forceinline__ f32x2 mul_add2(f32x2 a, f32x2 b, f32x2 s, f32x2 one) { return add2(s, mul2(a, b), one); }  // s + a*b, each rounded

constexpr int kST = 64;   // tokens per CTA of the score kernel
constexpr int kSP = 128;  // positions per CTA of the score kernel
constexpr int kSC = 32;   // columns of a stage

// grid (position tiles, token tiles, heads), 256 threads. Warp w owns tokens 8w..8w+7 of the tile, its lane l positions 2l, 2l+1,
// 64+2l, 65+2l: two position pairs, whose keys lie interleaved in shared memory, against eight queries, which lie there with every
// value twice, so that both operands of a packed instruction are loaded as they are (made twice in registers, a quarter of what
// the FP32 pipe issued were moves). Bound by that pipe, 79 % busy, 70 % of the load unit. The columns come in stages of 32, two in
// shared memory and the next on its way in registers: rows of all columns left one warp in four of what fits, and took longer
// than the moves had. us of the four 512-token pieces of a 1999-token prompt (4x4 patches with moves / this): 56 141 226 309 /
// 61 140 218 277.
template <int HD>
__global__ void __launch_bounds__(256, 2) tile_scores_kernel(const float *__restrict__ q, const float *__restrict__ kc, float *__restrict__ scores,
                                                             int n_head, int n_head_kv, const int32_t *__restrict__ meta, int max_kv, int ntok,
                                                             f32x2 one) {
    constexpr int S = 2 * kSC + 4;  // row stride: 16-byte aligned, neighbouring rows in different bank groups
    constexpr int C4 = kSC / 4, kStage = (kST + kSP / 2) * S;
    extern __shared__ __align__(16) float sm[];
    __shared__ int s_pos[kST];
    pdl_trigger();
    pdl_wait();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int p0 = blockIdx.x * kSP, t0 = blockIdx.y * kST, h = blockIdx.z;
    if (tid < kST) s_pos[tid] = (t0 + tid < ntok) ? meta[2 * (t0 + tid) + 1] : -1;
    __syncthreads();
    int maxpos = -1;
    for (int i = 0; i < kST; i++) maxpos = max(maxpos, s_pos[i]);
    if (p0 > maxpos) return;
    int wpos = -1;  // the last position of this warp's tokens: in front of the tile (or no tokens left), it only brings its share
    for (int i = 0; i < 8; i++) wpos = max(wpos, s_pos[8 * warp + i]);
    const int kv_dim = n_head_kv * HD;
    // What this thread brings of a stage: rows tid / 8 and 32 further of the position pairs, the same rows of the queries, four
    // columns of each. (A position past the last scores like the last one, a token past the end likewise; neither is stored.)
    const int r = tid / C4, c = tid % C4;
    const float *kh = kc + (size_t)(h / (n_head / n_head_kv)) * HD + 4 * c, *qh = q + (size_t)h * HD + 4 * c;
    const float *src[6];
#pragma unroll
    for (int u = 0; u < 2; u++) {
        const int p = p0 + 2 * (r + 32 * u);
        src[3 * u] = kh + (size_t)min(p, maxpos) * kv_dim;
        src[3 * u + 1] = kh + (size_t)min(p + 1, maxpos) * kv_dim;
        src[3 * u + 2] = qh + (size_t)min(t0 + r + 32 * u, ntok - 1) * n_head * HD;
    }
    float4 in[6];
    auto load = [&](int s) {
#pragma unroll
        for (int u = 0; u < 6; u++) in[u] = *reinterpret_cast<const float4 *>(src[u] + s * kSC);
    };
    auto store = [&](int s) {
        float *sQ = sm + (s & 1) * kStage, *sK = sQ + kST * S;
#pragma unroll
        for (int u = 0; u < 2; u++) {
            const float4 a = in[3 * u], b = in[3 * u + 1], x = in[3 * u + 2];
            float4 *k = reinterpret_cast<float4 *>(sK + (r + 32 * u) * S + 8 * c), *d = reinterpret_cast<float4 *>(sQ + (r + 32 * u) * S + 8 * c);
            k[0] = make_float4(a.x, b.x, a.y, b.y);
            k[1] = make_float4(a.z, b.z, a.w, b.w);
            d[0] = make_float4(x.x, x.x, x.y, x.y);
            d[1] = make_float4(x.z, x.z, x.w, x.w);
        }
    };
    f32x2 acc[8][2];
#pragma unroll
    for (int i = 0; i < 8; i++) acc[i][0] = acc[i][1] = 0ull;
    load(0);
    store(0);
    __syncthreads();
#pragma unroll 1
    for (int s = 0; s < HD / kSC; s++) {
        if (s + 1 < HD / kSC) load(s + 1);
        const float *qb = sm + (s & 1) * kStage + (warp * 8) * S, *kb = sm + (s & 1) * kStage + (kST + lane) * S;
        if (p0 <= wpos) {
#pragma unroll 4
            for (int d2 = 0; d2 < kSC / 2; d2++) {  // two columns at a time
                ulonglong2 b[2];
#pragma unroll
                for (int j = 0; j < 2; j++) b[j] = *reinterpret_cast<const ulonglong2 *>(kb + j * 32 * S + 4 * d2);
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    const ulonglong2 a = *reinterpret_cast<const ulonglong2 *>(qb + i * S + 4 * d2);
#pragma unroll
                    for (int j = 0; j < 2; j++) acc[i][j] = mul_add2(a.y, b[j].y, mul_add2(a.x, b[j].x, acc[i][j], one), one);
                }
            }
        }
        if (s + 1 < HD / kSC) {
            store(s + 1);  // (the last readers of these rows passed the barrier in front of this stage)
            __syncthreads();
        }
    }
    const float scale = __fdiv_rn(1.0f, __fsqrt_rn((float)HD));
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const int t = t0 + warp * 8 + i, pos = s_pos[warp * 8 + i];
        float *row = scores + ((size_t)t * n_head + h) * max_kv;
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const int p = p0 + 64 * j + 2 * lane;
            const float2 v = unpack2(acc[i][j]), l = make_float2(__fmul_rn(v.x, scale), __fmul_rn(v.y, scale));
            if (p < pos) *reinterpret_cast<float2 *>(row + p) = l;
            else if (p == pos) row[p] = l.x;
        }
    }
}

// One warp per (token, head) row: the logits become the softmax weights e*inv in place. The rows' sums are walked side by
// side by the first warp, a lane per row (a warp per chain is one lane's adds at a whole warp's issue): with a warp per chain a
// prompt of 1999 tokens took 0.5 % longer. Bound by the issue of the exponentials and by latency (three CTAs of rows fill the shared
// memory): four positions a lane at a time instead of one, with the shorter exponential, took the four
// pieces of a 1999-token prompt from 35 65 98 140 to 28 50 75 102 us.
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
    // (four positions a lane at a time; rows are whole 16-byte pieces, and what lies beyond the row's positions counts for nothing)
    float lmax = -INFINITY;
    for (int p = 4 * lane; p < n; p += 128) {
        float4 l = *reinterpret_cast<const float4 *>(g + p);
        if (p + 1 >= n) l.y = -INFINITY;
        if (p + 2 >= n) l.z = -INFINITY;
        if (p + 3 >= n) l.w = -INFINITY;
        *reinterpret_cast<float4 *>(sl + p) = l;
        lmax = fmaxf(fmaxf(fmaxf(l.x, l.y), fmaxf(l.z, l.w)), lmax);
    }
    for (int off = 16; off > 0; off >>= 1) lmax = fmaxf(lmax, __shfl_xor_sync(0xffffffffu, lmax, off));
    for (int p = 4 * lane; p < n; p += 128) {
        float4 *l = reinterpret_cast<float4 *>(sl + p);
        float e[4] = {l->x, l->y, l->z, l->w};
        ref_expf4(e, lmax);
        *l = make_float4(e[0], e[1], e[2], e[3]);
    }
    __syncthreads();
    if (warp == 0 && lane < warps) {
        const int r = blockIdx.x * warps + lane;
        if (r < rows) s_inv[lane] = __fdiv_rn(1.0f, chain_sum(sm + (size_t)lane * n_cap, min(meta[2 * (r / n_head) + 1] + 1, n_cap), 0.0f));
    }
    __syncthreads();
    const float inv = s_inv[warp];
    for (int p = 4 * lane; p < n; p += 128) {
        const float4 e = *reinterpret_cast<const float4 *>(sl + p);
        *reinterpret_cast<float4 *>(g + p) = make_float4(__fmul_rn(e.x, inv), __fmul_rn(e.y, inv), __fmul_rn(e.z, inv), __fmul_rn(e.w, inv));
    }
}

constexpr int kOT = 16;  // tokens per CTA of the output kernel
constexpr int kOP = 16;  // positions per staged tile
constexpr int kWS = kOP + 4;

// grid (heads, token tiles), HD threads. Thread (ty, tx) = (tid / (HD/4), tid % (HD/4)) owns tokens 4ty..4ty+3 and the output
// columns 4tx..4tx+3. Bound by the FP32 pipe, 82 % busy while a CTA is there. A CTA is one warp per scheduler and 16 tokens: the
// 1024 CTAs of a 512-token piece are seven to an SM, all at once, and 99 % of that many; with two warps to a CTA a scheduler
// got three or four of them, with 32 tokens an SM three or four CTAs, and the others waited a fifth of the time. The longest tokens
// of all heads start first. us of the four pieces of a 1999-token prompt (32 tokens, 4x8 patches / this): 72 161 251 332 /
// 54 136 218 289.
template <int HD>
__global__ void __launch_bounds__(HD) tile_pv_kernel(const float *__restrict__ w, const float *__restrict__ vc, float *__restrict__ out, int n_head,
                                                     int n_head_kv, const int32_t *__restrict__ meta, int max_kv, int ntok, f32x2 one) {
    constexpr int HD4 = HD / 4;
    __shared__ __align__(16) float sW[3][kOT][kWS];
    __shared__ __align__(16) float sV[3][kOP][HD];
    __shared__ int s_pos[kOT];
    pdl_trigger();
    pdl_wait();
    const int tid = threadIdx.x, ty = tid / HD4, tx = tid % HD4;
    const int t0 = ((int)gridDim.y - 1 - (int)blockIdx.y) * kOT, h = blockIdx.x;  // the longest tiles start first
    if (tid < kOT) s_pos[tid] = (t0 + tid < ntok) ? meta[2 * (t0 + tid) + 1] : -1;
    __syncthreads();
    int maxpos = -1;
    for (int i = 0; i < kOT; i++) maxpos = max(maxpos, s_pos[i]);
    const int kv_dim = n_head_kv * HD, kvh = h / (n_head / n_head_kv);
    const float *vb = vc + (size_t)kvh * HD + 4 * tx;
    const int wr = (tid >> 2) % kOT, wp = 4 * (tid & 3), wpos = s_pos[wr];  // four weights of a stage: token wr, positions wp..
    const float *wrow = w + ((size_t)min(t0 + wr, ntok - 1) * n_head + h) * max_kv + wp;
    auto stage = [&](int pt, int buf) {
        if (tid < 4 * kOT) {
            const int valid = max(0, min(4, wpos - (pt * kOP + wp) + 1));
            cp_async16(&sW[buf][wr][wp], valid ? wrow + pt * kOP : w, 4 * valid);
        }
#pragma unroll
        for (int u = 0; u < kOP / 4; u++) {
            const int r = ty + 4 * u, p = pt * kOP + r;
            cp_async16(&sV[buf][r][4 * tx], vb + (size_t)min(p, maxpos) * kv_dim, p <= maxpos ? 16 : 0);
        }
    };
    f32x2 acc[4][2];
#pragma unroll
    for (int i = 0; i < 4; i++) acc[i][0] = acc[i][1] = 0ull;
    const int n_pt = maxpos / kOP + 1;  // maxpos >= 0: the tile holds at least one token
    stage(0, 0);
    cp_async_commit();
    if (n_pt > 1) stage(1, 1);
    cp_async_commit();
    for (int pt = 0, buf = 0; pt < n_pt; pt++, buf = buf == 2 ? 0 : buf + 1) {
        cp_async_wait<1>();
        __syncthreads();  // stage pt is there, and everyone is done with stage pt - 1, whose place stage pt + 2 takes
        if (pt + 2 < n_pt) stage(pt + 2, buf == 0 ? 2 : buf - 1);
        cp_async_commit();
#pragma unroll
        for (int p4 = 0; p4 < kOP / 4; p4++) {
            float4 wv[4];
#pragma unroll
            for (int i = 0; i < 4; i++) wv[i] = *reinterpret_cast<const float4 *>(&sW[buf][ty * 4 + i][4 * p4]);
#pragma unroll
            for (int c = 0; c < 4; c++) {
                const ulonglong2 v = *reinterpret_cast<const ulonglong2 *>(&sV[buf][4 * p4 + c][4 * tx]);
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const float wi = c == 0 ? wv[i].x : c == 1 ? wv[i].y : c == 2 ? wv[i].z : wv[i].w;
                    const f32x2 ww = pack2(wi, wi);
                    acc[i][0] = mul_add2(ww, v.x, acc[i][0], one);
                    acc[i][1] = mul_add2(ww, v.y, acc[i][1], one);
                }
            }
        }
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int t = t0 + ty * 4 + i;
        if (t < ntok) *reinterpret_cast<ulonglong2 *>(out + ((size_t)t * n_head + h) * HD + 4 * tx) = make_ulonglong2(acc[i][0], acc[i][1]);
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
    constexpr size_t smem_s = 2 * (kST + kSP / 2) * (2 * kSC + 4) * sizeof(float);
    static bool conf_s = false;
    if (!conf_s)
        conf_s = cudaFuncSetAttribute(tile_scores_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_s) == cudaSuccess &&
                 cudaFuncSetAttribute(tile_scores_kernel<128>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_s) == cudaSuccess;
    launch_k("tile_scores", hd == 64 ? tile_scores_kernel<64> : tile_scores_kernel<128>, dim3((n_kv_max + kSP - 1) / kSP, (ntok + kST - 1) / kST, n_head),
             dim3(256), smem_s, q, kc, scores, n_head, n_head_kv, meta, max_kv, ntok, kOne2);
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
    const dim3 grid(n_head, (ntok + kOT - 1) / kOT);
    if (hd == 64)
        launch_k("tile_pv", tile_pv_kernel<64>, grid, dim3(hd), 0, (const float *)scores, vc, out, n_head, n_head_kv, meta, max_kv, ntok, kOne2);
    else
        launch_k("tile_pv", tile_pv_kernel<128>, grid, dim3(hd), 0, (const float *)scores, vc, out, n_head, n_head_kv, meta, max_kv, ntok, kOne2);
}
}
