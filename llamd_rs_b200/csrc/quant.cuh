// Device helpers shared by the quantizing kernels: the exponential, the Q8_K
// block quantizer and SiLU(gate)*up, each in the reference's operation order.
#pragma once
#include "common.cuh"

namespace llamd {

// The reference calls Rust's f32::exp, i.e. the host libm's expf. Here the exponential is evaluated in double and
// rounded once to f32, which is the correctly rounded result; the host's expf is not always (glibc's differs by one
// ulp on roughly one input in 12000). Routing decisions and Q8_K roundings downstream amplify such a bit, so the
// library makes the two agree exactly: when it starts it evaluates this very expression on the device for EVERY
// float in the range where exp is neither 1, 0 nor infinite, compares with the host's expf, and keeps the inputs
// that differ in a hash table (runtime.cu: build_exp_table). ref_expf looks its argument up there: one probe of a
// sparsely filled table in L2, a hit only for the listed inputs. Each translation unit has its own copy of the two
// pointers (constant memory), set through the binder it registers below.
static __constant__ const uint32_t *c_exp_keys = nullptr;  // [mask + 1] input bit patterns, 0 = empty slot
static __constant__ const uint32_t *c_exp_vals = nullptr;  // [mask + 1] the host expf's result bits
static __constant__ uint32_t c_exp_mask = 0;
static __constant__ uint32_t c_exp_window = 0;  // see exp_needs_lookup; 0 = look every input up

// The host's expf can differ from the correctly rounded value only where exp(x) lies very close to the midpoint of
// two neighbouring floats (its error before the final rounding is a few thousandths of an ulp). The 29 bits of the
// double result below float precision say how close: the table is consulted only within `window` (in units of
// 2^-29 ulp) of the midpoint. The window is measured when the table is built: the largest distance over every listed
// input, on the device, plus one; an input outside it is therefore not in the table. Results that are subnormal as
// floats round at another bit position and are always looked up.
__device__ __forceinline__ bool exp_needs_lookup(float x, double yd, uint32_t window) {
    if (window == 0 || x < -87.0f) return true;
    const uint32_t frac = (uint32_t)__double_as_longlong(yd) & 0x1FFFFFFFu;
    return frac - (0x10000000u - window) < 2u * window;  // |frac - 2^28| < window
}

// e^x in double for a float x: x = k ln2 + r with k = round(x / ln2), taken by the rounding of an addition, ln2 in two parts
// (Cody and Waite), for e^r the polynomial of degree 10 that equals it at the eleven Chebyshev nodes of |r| <= ln2 / 2 (relative
// error 3.3e-16; evaluated in double 4.6e-16, two units in the last place of a double, where CUDA's exp((double)x) has one), and k
// into the exponent, in half its instructions. The result is rounded to f32 behind it, and the table below is made with this very
// function, so that every float's result is the host's all the same. Inputs whose float result is 0 or
// infinite are cut to where it still is; a NaN comes out as one.
__device__ __forceinline__ double exp_f64(float x) {
    x = x < -110.0f ? -110.0f : x > 100.0f ? 100.0f : x;
    const double xd = (double)x, shift = 6755399441055744.0;  // 1.5 * 2^52: the sum's last place is 1
    const double t = __fma_rn(xd, 1.4426950408889634, shift), k = __dsub_rn(t, shift);
    const double r = __fma_rn(k, -5.497923018708371e-14, __fma_rn(k, -0.6931471805598903, xd));  // (the first part has 42 bits: k times it is exact)
    double p = __fma_rn(r, 2.762635725527078e-07, 2.7640180812804505e-06);
    p = __fma_rn(p, r, 2.480150434696448e-05);
    p = __fma_rn(p, r, 0.00019841170270400204);
    p = __fma_rn(p, r, 0.0013888888932488625);
    p = __fma_rn(p, r, 0.008333333385667814);
    p = __fma_rn(p, r, 0.04166666666657314);
    p = __fma_rn(p, r, 0.16666666666554406);
    p = __fma_rn(p, r, 0.5000000000000006);
    p = __fma_rn(p, r, 1.0000000000000067);
    p = __fma_rn(p, r, 1.0);
    return __hiloint2double(__double2hiint(p) + (__double2loint(t) << 20), __double2loint(p));
}

__device__ __forceinline__ float exp_exception(float x, float y) {  // the listed result for x, or y
    const uint32_t *keys = c_exp_keys;
    const uint32_t b = __float_as_uint(x), mask = c_exp_mask;
    uint32_t h = (b * 2654435761u) >> 8 & mask;
    for (int probe = 0; probe < 64; probe++) {  // (a table at most a quarter full: runs are short)
        const uint32_t k = __ldg(keys + h);
        if (k == 0) break;
        if (k == b) return __uint_as_float(__ldg(c_exp_vals + h));
        h = (h + 1) & mask;
    }
    return y;
}

__device__ __forceinline__ float ref_expf(float x) {
    const double yd = exp_f64(x);
    const float y = __double2float_rn(yd);
    return c_exp_keys && exp_needs_lookup(x, yd, c_exp_window) ? exp_exception(x, y) : y;
}

// v[i] = ref_expf(v[i] - m): four side by side, and one branch for all of their exceptions
__device__ __forceinline__ void ref_expf4(float v[4], float m) {
    float y[4];
    bool look[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        v[i] = __fsub_rn(v[i], m);
        const double yd = exp_f64(v[i]);
        y[i] = __double2float_rn(yd);
        look[i] = exp_needs_lookup(v[i], yd, c_exp_window);
    }
    if (c_exp_keys && (look[0] || look[1] || look[2] || look[3])) {
#pragma unroll
        for (int i = 0; i < 4; i++)
            if (look[i]) y[i] = exp_exception(v[i], y[i]);
    }
#pragma unroll
    for (int i = 0; i < 4; i++) v[i] = y[i];
}

void register_exp_binder(void (*bind)(const uint32_t *, const uint32_t *, uint32_t, uint32_t));
namespace {
inline void bind_exp_table_here(const uint32_t *keys, const uint32_t *vals, uint32_t mask, uint32_t window) {
    cudaMemcpyToSymbol(c_exp_keys, &keys, sizeof keys);
    cudaMemcpyToSymbol(c_exp_vals, &vals, sizeof vals);
    cudaMemcpyToSymbol(c_exp_mask, &mask, sizeof mask);
    cudaMemcpyToSymbol(c_exp_window, &window, sizeof window);
}
struct ExpBinderRegistration {
    ExpBinderRegistration() { register_exp_binder(bind_exp_table_here); }
};
static ExpBinderRegistration s_exp_binder_registration;
}  // namespace

// ---- Q8_K: crates/llamd-quant/src/dot.rs:88-128 ---------------------------
// One warp per 256-element block; lane l owns elements 8l..8l+7.
// Produces qs[256] (natural order), d and optionally bsums[16], and optionally the quants in the GEMMs' operand order as well
// (t32_place, t32_element in q6k_layout.cuh): lane l holds byte k of word l / 4 of every residue, where k swaps the two bits
// of l % 4. (A launch of its own for that order cost 3 to 4 us four times a layer.)
__device__ __forceinline__ void q8k_quantize_block(const float v[8], int lane, int8_t *__restrict__ qs, float *__restrict__ d_out,
                                                   int16_t *__restrict__ bsums, int8_t *__restrict__ rm = nullptr) {
    // the SIGNED value at the largest magnitude, first such element
    float amax = 0.0f, mx = 0.0f;
    int idx = 0;
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const float a = fabsf(v[i]);
        if (a > amax) {
            amax = a;
            mx = v[i];
            idx = lane * 8 + i;
        }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        const float oa = __shfl_xor_sync(0xffffffffu, amax, off);
        const float om = __shfl_xor_sync(0xffffffffu, mx, off);
        const int oi = __shfl_xor_sync(0xffffffffu, idx, off);
        if (oa > amax || (oa == amax && oi < idx)) {
            amax = oa;
            mx = om;
            idx = oi;
        }
    }
    int q[8];
    float dd = 0.0f;
    if (amax == 0.0f) {
#pragma unroll
        for (int i = 0; i < 8; i++) q[i] = 0;
    } else {
        const float iscale = __fdiv_rn(-127.0f, mx);
#pragma unroll
        for (int i = 0; i < 8; i++) q[i] = min(127, __float2int_rn(__fmul_rn(iscale, v[i])));
        dd = __fdiv_rn(1.0f, iscale);
    }
    uint32_t w0 = 0, w1 = 0;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        w0 |= ((uint32_t)q[i] & 0xFFu) << (8 * i);
        w1 |= ((uint32_t)q[4 + i] & 0xFFu) << (8 * i);
    }
    *reinterpret_cast<uint2 *>(qs + lane * 8) = make_uint2(w0, w1);
    if (rm) {
#pragma unroll
        for (int i = 0; i < 8; i++)
            rm[64 * (i >> 1) + 16 * ((lane >> 2) & 3) + 8 * (i & 1) + 4 * (lane >> 4) + 2 * (lane & 1) + ((lane >> 1) & 1)] = (int8_t)q[i];
    }
    if (lane == 0) *d_out = dd;
    if (bsums) {
        int s = 0;
#pragma unroll
        for (int i = 0; i < 8; i++) s += q[i];
        s += __shfl_xor_sync(0xffffffffu, s, 1);
        if ((lane & 1) == 0) bsums[lane >> 1] = (int16_t)s;
    }
}

// silu(gate) * up (crates/llamd-cpu/src/lib.rs:103-114, layer.rs:252):
// v / (1 + exp(-v)), then the elementwise product.
__device__ __forceinline__ float silu_mul(float g, float u) {
    const float s = __fdiv_rn(g, __fadd_rn(1.0f, ref_expf(-g)));
    return __fmul_rn(s, u);
}

}  // namespace llamd
