// out[t][row] = fold(-0.0, +) of w[row][i] * x[t][i], i ascending: the f32 matvec of
// crates/llamd-models/src/model.rs:253-263 for the ntok tokens of a prefill tile at once.
//
// The sum over i is one chain per output element and stays one: a lane owns a row and walks i in order for two or four
// tokens whose chains take turns. 2048 dependent adds are 4.6 us at 1.9 GHz whatever else happens, so everything else has
// to fit beside them: the copies of the operands (chunks of 128 columns, 4 or 5 in flight, by warps of their own, the
// weights' first ones before the dependency wait where the caller says that no launch in front writes them), the shared loads and the multiplies (a register set ahead of the adds).
// Bound by instruction issue of the adding warps, and by L2 for many tokens. The router logits of a tile (128 experts x
// 2048 columns) are the user, us with a 2x2 patch of chains per thread (16 tokens a CTA, one 64-column chunk ahead) / now:
// 8 to 64 tokens 36.7 / 14.6, 128 36.7 / 21, 512 37.5 / 24.6, 2000 83 / 84.
#include "common.cuh"

namespace llamd {
namespace {

__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

constexpr int kFR = 32;       // rows per CTA: a lane each
constexpr int kFLoaders = 2;  // warps that copy
constexpr int kFK = 128;      // columns per staged chunk
constexpr int kFS = kFK + 4;  // shared-memory row stride: 16-byte aligned, neighbouring rows in different bank groups

// grid (row tiles, token tiles). Adding warp v owns tokens TPW*v .. +TPW-1 of its CTA's tile, lane r row r.
template <int TPW, int kFWarps, int kFStages>
__global__ void __launch_bounds__(32 * (kFWarps + kFLoaders)) matmul_f32_tokens_kernel(const float *__restrict__ w, const float *__restrict__ x, float *__restrict__ out,
                                                                         int k, int rows, int ntok, int w_ready) {
    constexpr int kTok = TPW * kFWarps;
    extern __shared__ __align__(16) float sm[];  // [kFStages][kFR + kTok][kFS]
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int r0 = blockIdx.x * kFR, t0 = blockIdx.y * kTok;
    const int n_chunks = (k + kFK - 1) / kFK;
    pdl_trigger();
    if (warp >= kFWarps) {
        // ---- loaders: 16-byte pieces, a warp takes whole rows of 32; what lies outside the matrix is left out (never read).
        // (Copying on the side, the adding warps spent half their time on the copies' addresses.)
        const int v = warp - kFWarps;
        auto rows_of = [&](int ch, const float *src, int n, int first) {
            const uint32_t dst = (uint32_t)__cvta_generic_to_shared(sm + ((ch % kFStages) * (kFR + kTok) + first) * kFS + 4 * lane);
            if (ch * kFK + 4 * lane >= k) return;
            const float *p = src + ch * kFK + 4 * lane;
#pragma unroll 4
            for (int r = v; r < n; r += kFLoaders)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + r * kFS * 4), "l"(p + (size_t)r * k) : "memory");
        };
        const float *ws = w + (size_t)r0 * k, *xs = x + (size_t)t0 * k;
        const int nw = min(kFR, rows - r0), nx = min(kTok, ntok - t0);
        if (!w_ready) pdl_wait();
        for (int ch = 0; ch < kFStages - 1 && ch < n_chunks; ch++) rows_of(ch, ws, nw, 0);
        if (w_ready) pdl_wait();
        for (int ch = 0; ch < kFStages - 1; ch++) {
            if (ch < n_chunks) rows_of(ch, xs, nx, kFR);
            cp_async_commit();  // (the weights above join the first group)
        }
        for (int ch = 0; ch < n_chunks; ch++) {
            cp_async_wait<kFStages - 2>();
            __syncthreads();
            if (ch + kFStages - 1 < n_chunks) rows_of(ch + kFStages - 1, ws, nw, 0), rows_of(ch + kFStages - 1, xs, nx, kFR);
            cp_async_commit();
        }
        return;
    }
    pdl_wait();
    float acc[TPW];
#pragma unroll
    for (int i = 0; i < TPW; i++) acc[i] = -0.0f;
    const bool live = t0 + TPW * warp < ntok;  // (uniform over the warp)
    for (int ch = 0; ch < n_chunks; ch++) {
        __syncthreads();  // (chunk ch has landed; and everyone is done with the chunk whose place the next one takes)
        if (!live) continue;
        const float *base = sm + (ch % kFStages) * (kFR + kTok) * kFS;
        const float4 *wr = reinterpret_cast<const float4 *>(base + lane * kFS);
        const float4 *xr = reinterpret_cast<const float4 *>(base + (kFR + TPW * warp) * kFS);
        const int n4 = min(kFK, k - ch * kFK) >> 2;  // no padding terms: a chain holds exactly its k products
        if (n4 == kFK / 4) {
            // eight columns a half-step: two register sets alternate, a set is loaded again right after its products are
            // formed, and the products of one set are formed among the adds of the other's
            constexpr int G = 2;
            const uint32_t wa = (uint32_t)__cvta_generic_to_shared(wr), xa = (uint32_t)__cvta_generic_to_shared(xr);
            float4 w0[G], x0[TPW][G], w1[G], x1[TPW][G], p0[TPW][G], p1[TPW][G];
            auto fetch = [&](int c, float4 (&wv)[G], float4 (&xv)[TPW][G]) {
#pragma unroll
                for (int g = 0; g < G; g++) {
                    wv[g] = chain_lds(wa + 16 * (c + g));
#pragma unroll
                    for (int i = 0; i < TPW; i++) xv[i][g] = chain_lds(xa + 4 * kFS * i + 16 * (c + g));
                }
            };
            auto products = [&](const float4 (&wv)[G], const float4 (&xv)[TPW][G], float4 (&o)[TPW][G]) {
#pragma unroll
                for (int i = 0; i < TPW; i++)
#pragma unroll
                    for (int g = 0; g < G; g++)
                        o[i][g] = make_float4(__fmul_rn(wv[g].x, xv[i][g].x), __fmul_rn(wv[g].y, xv[i][g].y), __fmul_rn(wv[g].z, xv[i][g].z),
                                              __fmul_rn(wv[g].w, xv[i][g].w));
            };
            auto add = [&](const float4 (&o)[TPW][G]) {  // (the tokens' chains take turns)
#pragma unroll
                for (int e = 0; e < 4 * G; e++)
#pragma unroll
                    for (int i = 0; i < TPW; i++) acc[i] = __fadd_rn(acc[i], (&o[i][e >> 2].x)[e & 3]);
            };
            fetch(0, w0, x0);
            fetch(G, w1, x1);
            products(w0, x0, p0);
            fetch(2 * G, w0, x0);
#pragma unroll 1
            for (int c = 0; c < kFK / 4; c += 2 * G) {
                products(w1, x1, p1);
                fetch(c + 3 * G, w1, x1);
                add(p0);
                products(w0, x0, p0);
                fetch(c + 4 * G, w0, x0);  // (the last of them lie in the next stage or the padding behind the last: never used)
                add(p1);
            }
        } else {
            for (int c = 0; c < n4; c++) {
                const float4 a = wr[c];
#pragma unroll
                for (int i = 0; i < TPW; i++) {
                    const float4 b = xr[i * (kFS / 4) + c];
                    acc[i] = __fadd_rn(acc[i], __fmul_rn(a.x, b.x));
                    acc[i] = __fadd_rn(acc[i], __fmul_rn(a.y, b.y));
                    acc[i] = __fadd_rn(acc[i], __fmul_rn(a.z, b.z));
                    acc[i] = __fadd_rn(acc[i], __fmul_rn(a.w, b.w));
                }
            }
        }
    }
    if (r0 + lane < rows) {
#pragma unroll
        for (int i = 0; i < TPW; i++) {
            const int t = t0 + TPW * warp + i;
            if (t < ntok) out[(size_t)t * rows + r0 + lane] = acc[i];
        }
    }
}

template <int TPW, int kFWarps, int kFStages>
void matmul_f32_tokens_launch(const float *w, const float *x, float *out, int k, int rows, int ntok, bool w_ready) {
    constexpr int kTok = TPW * kFWarps, kSmem = kFStages * (kFR + kTok) * kFS * 4 + 256;  // (+ what the last loads run past)
    static bool configured = false;
    if (!configured) {
        if (cudaFuncSetAttribute(matmul_f32_tokens_kernel<TPW, kFWarps, kFStages>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem) != cudaSuccess) {
            set_error(cudaGetLastError(), "matmul_f32_tokens smem attribute");
            return;
        }
        configured = true;
    }
    launch_kc(PDL_ROUTER, "matmul_f32_tokens", matmul_f32_tokens_kernel<TPW, kFWarps, kFStages>, dim3((rows + kFR - 1) / kFR, (ntok + kTok - 1) / kTok), dim3(32 * (kFWarps + kFLoaders)), kSmem,
              w, x, out, k, rows, ntok, (int)w_ready);
}

}  // namespace
}  // namespace llamd

using namespace llamd;

void llamd::matmul_f32_tokens(const float *w, const float *x, float *out, int k, int rows, int ntok, bool w_ready) {
    if (ntok <= 0 || rows <= 0) return;
    if (k < 4 || k % 4) {
        set_error_msg("matmul_f32_tokens: k must be a positive multiple of 4");
        return;
    }
    // Few tokens: two warps of two tokens, so that a warp has nearly an SM to itself. More: four of four, or the CTAs' reads of
    // the matrix become the limit (2048 columns of 32 rows each: 128 tokens 21 us this way and 24 that, 512 tokens 33 and 25).
    // Five chunks in flight fill an SM with one such CTA; four let two share it, which is worth it only once there are more
    // CTAs than SMs (2000 tokens 96 and 84 us, but 300 tokens 24 and 37: two on some SMs, none on others).
    const long long ctas = (long long)((rows + kFR - 1) / kFR) * ((ntok + 15) / 16);
    if (ntok <= 128)
        matmul_f32_tokens_launch<2, 2, 5>(w, x, out, k, rows, ntok, w_ready);
    else if (ctas <= 148)
        matmul_f32_tokens_launch<4, 4, 5>(w, x, out, k, rows, ntok, w_ready);
    else
        matmul_f32_tokens_launch<4, 4, 4>(w, x, out, k, rows, ntok, w_ready);
}
extern "C" void llamd_fwd_matmul_f32_tokens(const float *w, const float *x, float *out, int k, int rows, int ntok) {
    matmul_f32_tokens(w, x, out, k, rows, ntok, false);
}
