// out[t][row] = fold(-0.0, +) of w[row][i] * x[t][i], i ascending: the f32 matvec of
// crates/llamd-models/src/model.rs:253-263 for the ntok tokens of a prefill tile at once.
//
// The sum over i is one chain per output element and stays one: a lane owns a row and walks i in order for two or four
// tokens whose chains take turns. 2048 dependent adds are 4.6 us at 1.9 GHz whatever else happens, so everything else has
// to fit beside them: the copies of the operands (chunks of 128 columns, 4 or 5 in flight, by warps of their own, the
// weights' first ones before the dependency wait where the caller says that no launch in front writes them), the shared loads and the multiplies (a register set ahead of the adds).
// Bound by instruction issue of the adding warps, and by L2 for many tokens; where the CTAs are more than two per SM a 2x2
// patch of chains per thread is quicker (matmul_f32_patch_kernel). The router logits of a tile (128 experts x 2048 columns) are
// the user, us with patches / this: 8 to 64 tokens 37.0 / 15 to 18, 128 37.0 / 22.9, 512 37.0 / 25.0, 1000 53.4 / 44.4, 2000 80.1 / 85.3.
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

// The same for many CTAs: a thread owns a 2x2 patch of outputs (two tokens x two rows) and walks i in order for its four
// accumulators; a CTA stages 64 columns of 16 tokens and 32 rows (double-buffered), every staged value feeds two chains. The copies
// and the multiplies stand between the adds, which costs a lone CTA twice the time; eight of them on an SM hide it.
// grid (row tiles, token tiles), 128 threads. Thread (ty, tx) = (tid / 16, tid % 16) owns tokens 2ty, 2ty+1 and rows tx, tx+16.
constexpr int kPT = 16, kPK = 64, kPS = kPK + 4;
__device__ __forceinline__ void cp_async16(void *dst, const void *src, int bytes) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(bytes) : "memory");
}
__global__ void __launch_bounds__(128) matmul_f32_patch_kernel(const float *__restrict__ w, const float *__restrict__ x, float *__restrict__ out, int k,
                                                               int rows, int ntok) {
    __shared__ __align__(16) float sX[2][kPT][kPS];
    __shared__ __align__(16) float sW[2][kFR][kPS];
    pdl_trigger();
    pdl_wait();
    const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
    const int r0 = blockIdx.x * kFR, t0 = blockIdx.y * kPT;
    auto stage = [&](int k0, int buf) {
        // 16-byte pieces: (16 + 32) rows x 16 pieces = 768, six per thread
        for (int idx = tid; idx < (kPT + kFR) * (kPK / 4); idx += 128) {
            const int r = idx >> 4, c = idx & 15;
            const int col = k0 + 4 * c;
            const int bytes = col < k ? 16 : 0;  // k is a multiple of 4
            if (r < kPT) {
                const int t = t0 + r;
                cp_async16(&sX[buf][r][4 * c], x + (size_t)min(t, ntok - 1) * k + min(col, k - 4), t < ntok ? bytes : 0);
            } else {
                const int row = r0 + r - kPT;
                cp_async16(&sW[buf][r - kPT][4 * c], w + (size_t)min(row, rows - 1) * k + min(col, k - 4), row < rows ? bytes : 0);
            }
        }
        cp_async_commit();
    };
    float acc[2][2] = {{-0.0f, -0.0f}, {-0.0f, -0.0f}};
    const int n_chunks = (k + kPK - 1) / kPK;
    stage(0, 0);
    for (int ch = 0; ch < n_chunks; ch++) {
        const int buf = ch & 1;
        if (ch + 1 < n_chunks) {
            stage((ch + 1) * kPK, buf ^ 1);
            cp_async_wait<1>();
        } else {
            cp_async_wait<0>();
        }
        __syncthreads();
        const int n4 = min(kPK, k - ch * kPK) >> 2;  // no padding terms: a chain holds exactly its k products
#pragma unroll 4
        for (int c4 = 0; c4 < n4; c4++) {
            float4 a[2], b[2];
#pragma unroll
            for (int i = 0; i < 2; i++) a[i] = *reinterpret_cast<const float4 *>(&sX[buf][2 * ty + i][4 * c4]);
#pragma unroll
            for (int j = 0; j < 2; j++) b[j] = *reinterpret_cast<const float4 *>(&sW[buf][tx + 16 * j][4 * c4]);
#pragma unroll
            for (int i = 0; i < 2; i++)
#pragma unroll
                for (int j = 0; j < 2; j++) {
                    float s = acc[i][j];
                    s = __fadd_rn(s, __fmul_rn(b[j].x, a[i].x));
                    s = __fadd_rn(s, __fmul_rn(b[j].y, a[i].y));
                    s = __fadd_rn(s, __fmul_rn(b[j].z, a[i].z));
                    s = __fadd_rn(s, __fmul_rn(b[j].w, a[i].w));
                    acc[i][j] = s;
                }
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 2; i++) {
        const int t = t0 + 2 * ty + i;
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const int row = r0 + tx + 16 * j;
            if (t < ntok && row < rows) out[(size_t)t * rows + row] = acc[i][j];
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
    // Small products: two warps of two tokens, so that a warp has nearly an SM to itself, while such CTAs are two per SM at most.
    // More: four of four, or the CTAs' reads of the matrix become the limit; five chunks in flight fill an SM with one such CTA,
    // four let two share it, which is worth it only once there are more CTAs than SMs. Beyond two of those per SM, the patches.
    // us at 2048 columns, two of two / four of four / patches: 128 rows, 128 tokens 22.9 / 24.8 / 37.0; 256 rows, 128 tokens 23.9 /
    // 24.9 / 37.0; 1024 rows, 64 tokens 43.9 / 25.1 / 37.0, 128 tokens 85 / 44 / 53; 300 tokens - / 104 / 98, 2000 - / 568 / 496.
    const int row_tiles = (rows + kFR - 1) / kFR;
    const long long small = (long long)row_tiles * ((ntok + 3) / 4), ctas = (long long)row_tiles * ((ntok + 15) / 16);
    if (small <= 2 * 148)
        matmul_f32_tokens_launch<2, 2, 5>(w, x, out, k, rows, ntok, w_ready);
    else if (ctas <= 148)
        matmul_f32_tokens_launch<4, 4, 5>(w, x, out, k, rows, ntok, w_ready);
    else if (ctas <= 2 * 148)
        matmul_f32_tokens_launch<4, 4, 4>(w, x, out, k, rows, ntok, w_ready);
    else
        launch_k("matmul_f32_patch", matmul_f32_patch_kernel, dim3(row_tiles, (ntok + kPT - 1) / kPT), dim3(128), 0, w, x, out, k, rows, ntok);
}
extern "C" void llamd_fwd_matmul_f32_tokens(const float *w, const float *x, float *out, int k, int rows, int ntok) {
    matmul_f32_tokens(w, x, out, k, rows, ntok, false);
}
