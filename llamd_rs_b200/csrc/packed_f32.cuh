// Two f32 values in one register pair: an instruction works on both, each rounded as its scalar form rounds it.
#pragma once

namespace llamd {

typedef unsigned long long f32x2;
constexpr f32x2 kOne2 = 0x3F8000003F800000ull;  // 1.0f twice; kernels get it as a parameter (see add2)

__device__ __forceinline__ f32x2 pack2(float a, float b) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float2 unpack2(f32x2 v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
// s + t, rounded once, as an fma with 1.0 in a value the compiler cannot see: a packed multiply feeding a packed add is
// contracted into one fma, which rounds once where the reference rounds twice.
__device__ __forceinline__ f32x2 add2(f32x2 s, f32x2 t, f32x2 one) { return fma2(t, one, s); }

}  // namespace llamd
