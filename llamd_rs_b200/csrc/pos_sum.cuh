// An ordered f32 sum of terms that are not negative, by a whole CTA, bit for bit what the chain s = s + p gives.
//
// The chain is bound by its own latency: 2048 dependent adds are 9100 cycles, in which the CTA's other threads wait (the two
// sums of squares of a layer, the softmax sum of a long context). But while s stays inside one binade its bit pattern k
// counts units in the last place, and adding p >= 0 adds to k an integer that depends on p and on k's parity alone: p / ulp
// rounded, where a tie goes to the even side. So any run of terms is a pair (increment if k is even, increment if k is odd),
// pairs of adjacent runs compose, and a run's pair can be formed before its start is known, given only the binade.
//   - thread 0 walks the first kHead terms as the chain that they are: the sum doubles five times among them;
//   - meanwhile the other warps sum all runs of 64 terms approximately, scan these sums to learn which binade the chain will
//     be in at each run, and form the runs' pairs: a thread per 8 terms, composed over 8 lanes;
//   - thread 0 goes on from run to run: where start and end lie in the binade that the pair was formed for, a run is one
//     integer addition, eight of them at a time speculatively; where not (the sum crosses a power of two there, or the
//     approximation was off) it takes the run's terms.
// Every use of a pair is checked against the exact running value, so a wrong guess costs time and never a bit; zeros,
// subnormals, infinities and NaNs always take the terms themselves.
// Measured, cycles, chain / this with 256 threads: 2048 terms 9100 / 5500, 4096 17500 / 8900 (12 %
// more with three CTAs on the SM).
#pragma once
#include "common.cuh"

namespace llamd {

constexpr int kPosSeg = 4096;  // terms per pass over the scratch below; a longer sum takes several
constexpr int kPosRuns = kPosSeg / 64;
struct PosScratch {
    float sum[kPosRuns];
    int4 run[kPosRuns + 8];  // (exponent in place, or -1; increment from even; what an odd start adds to it)
    uint32_t start;
};

__device__ __forceinline__ void pos_compose(int &e, int &o, int ge, int go) {
    e += (e & 1) ? go : ge;
    o += (o & 1) ? ge : go;
}

template <int NT>
__device__ __forceinline__ void pos_prep(const float *s, int len, PosScratch &sc, int head) {  // all warps but warp 0
    const int t = threadIdx.x - 32, lane = threadIdx.x & 31;
    auto load8 = [&](int t0, float (&v)[8]) {
#pragma unroll
        for (int h = 0; h < 2; h++) {
            float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
            const int i = t0 + 4 * h;
            if (i + 4 <= len) x = *reinterpret_cast<const float4 *>(s + i);
            else if (i < len) x = make_float4(s[i], i + 1 < len ? s[i + 1] : 0.f, i + 2 < len ? s[i + 2] : 0.f, 0.f);
            v[4 * h] = x.x, v[4 * h + 1] = x.y, v[4 * h + 2] = x.z, v[4 * h + 3] = x.w;
        }
    };
#pragma unroll 1
    for (int g = t; g < kPosSeg / 8; g += NT - 32) {
        float q = 0.0f;
        if ((g & ~31) * 8 < len) {  // (uniform over the warp)
            float v[8];
            load8(g * 8, v);
            q = ((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7]));
            q += __shfl_xor_sync(0xffffffffu, q, 1);
            q += __shfl_xor_sync(0xffffffffu, q, 2);
            q += __shfl_xor_sync(0xffffffffu, q, 4);
        }
        if ((lane & 7) == 0) sc.sum[g >> 3] = q;
    }
    asm volatile("bar.sync 1, %0;" ::"n"(NT - 32) : "memory");
    // every warp scans the runs' sums: lane = two runs
    const float2 two = reinterpret_cast<const float2 *>(sc.sum)[lane];
    float incl = two.x + two.y + (lane == 0 && !head ? __uint_as_float(sc.start) : 0.0f);
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const float x = __shfl_up_sync(0xffffffffu, incl, off);
        if (lane >= off) incl += x;
    }
#pragma unroll 1
    for (int g = t + head / 8; (g - lane) * 8 < len; g += NT - 32) {  // (the head's runs need no pairs)
        const int run = g >> 3;
        const float top = __shfl_sync(0xffffffffu, incl, (run >> 1) & 31), second = sc.sum[(run | 1) & (kPosRuns - 1)];
        const float b = (run & 1) ? top : top - second, a = b - sc.sum[run & (kPosRuns - 1)];  // the chain behind and before this run, about
        float v[8];
        load8(g * 8, v);
        int E = (int)(__float_as_uint(a) >> 23);
        if ((int)(__float_as_uint(b) >> 23) != E || E < 23 || E > 253) E = -1;
        const float scale = __uint_as_float((uint32_t)(277 - (E < 0 ? 127 : E)) << 23);  // 1 / ulp of that binade
        int e = 0, any = 0, r[8], tie[8];
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const float x = __fmul_rn(v[i], scale), y = __fadd_rn(x, 8388608.0f);  // y = 2^23 + x rounded to an integer
            r[i] = min((int)(__float_as_uint(y) - 0x4B000000u), 1 << 23);          // (a larger term leaves the binade anyway)
            const float d = __fsub_rn(x, __fsub_rn(y, 8388608.0f));
            tie[i] = fabsf(d) == 0.5f ? (d > 0.0f ? 1 : -1) : 0;                   // a tie: what an odd k adds besides
            any |= tie[i];
            e += r[i];
        }
        int o = e;
        if (any) {
            e = o = 0;
#pragma unroll
            for (int i = 0; i < 8; i++) pos_compose(e, o, r[i], r[i] + tie[i]);
        }
#pragma unroll
        for (int off = 1; off <= 4; off <<= 1) {  // (right in the lanes that count: multiples of 8 in the end)
            const int ge = __shfl_down_sync(0xffffffffu, e, off), go = __shfl_down_sync(0xffffffffu, o, off);
            pos_compose(e, o, ge, go);
        }
        if ((lane & 7) == 0 && run < kPosRuns) sc.run[run] = make_int4(E < 0 ? -1 : E << 23, e, o - e, 0);
    }
}

// s: shared memory, 16-byte aligned, n terms behind a barrier; all NT threads call it. The sum is thread 0's return value.
template <int NT>
__device__ __noinline__ float pos_chain_sum(const float *s, int n, PosScratch &sc) {
    constexpr int kHead = NT >= 256 ? 384 : 512;  // (about as long as the other warps' part takes)
    if (n <= 2 * kHead) return threadIdx.x == 0 ? chain_sum(s, n, 0.0f) : 0.0f;
    uint32_t bits = 0;
    for (int base = 0; base < n; base += kPosSeg, s += kPosSeg) {
        const int len = min(kPosSeg, n - base), head = base == 0 ? kHead : 0, runs = (len + 63) >> 6;
        if (threadIdx.x >= 32) pos_prep<NT>(s, len, sc, head);
        else if (threadIdx.x == 0 && head) bits = __float_as_uint(chain_sum(s, head, 0.0f));
        else if (threadIdx.x >= 24) sc.run[runs + threadIdx.x - 24].x = -1;  // (the speculation below reads past the last run)
        __syncthreads();
        if (threadIdx.x == 0) {
            for (int q = head >> 6; q < runs;) {
                int4 m[8];
#pragma unroll
                for (int i = 0; i < 8; i++) m[i] = sc.run[q + i];
                uint32_t k[9], bad = 0x100;
                k[0] = bits;
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    k[i + 1] = k[i] + (uint32_t)m[i].y + (k[i] & 1u) * (uint32_t)m[i].z;
                    const uint32_t eb = (uint32_t)m[i].x;
                    bad |= ((k[i] ^ eb) | (k[i + 1] ^ eb)) < (1u << 23) ? 0u : 1u << i;
                }
                const int good = __ffs((int)bad) - 1;
                bits = k[8];
#pragma unroll
                for (int i = 0; i < 8; i++) bits = good == i ? k[i] : bits;
                q += good;
                if (good < 8 && q < runs) {
                    bits = __float_as_uint(chain_sum(s + 64 * q, min(64, len - 64 * q), __uint_as_float(bits)));
                    q++;
                }
            }
            sc.start = bits;
        }
        if (base + kPosSeg < n) __syncthreads();
    }
    return __uint_as_float(bits);
}

}  // namespace llamd
