// Two FP32 values per 64-bit register: the packed arithmetic of sm_100
// (add, mul, fma .f32x2).  A packed operation rounds each half as the scalar
// one does and takes one issue slot for two results; the FP32 pipe's rate is
// the same (measured: 1.97 packed against 3.88 scalar fma per clock and SM).
#pragma once

#include <cuda_runtime.h>

namespace s2d {

typedef unsigned long long f2;  // rows r (low half) and r+1 (high half)

static __device__ __forceinline__ f2 pk(float lo, float hi) {
    f2 d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
    return d;
}
static __device__ __forceinline__ f2 dup(float v) { return pk(v, v); }
static __device__ __forceinline__ float lo(f2 v) {
    return __uint_as_float((unsigned)v);
}
static __device__ __forceinline__ float hi(f2 v) {
    return __uint_as_float((unsigned)(v >> 32));
}
static __device__ __forceinline__ f2 add2(f2 a, f2 b) {
    f2 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
static __device__ __forceinline__ f2 sub2(f2 a, f2 b) {
    f2 d;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
static __device__ __forceinline__ f2 mul2(f2 a, f2 b) {
    f2 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
static __device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
    f2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
// c0*d0 + c1*d1, one product rounded, then fused (the step kernels' dif)
static __device__ __forceinline__ f2 dif2(f2 c0, f2 d0, f2 c1, f2 d1) { return fma2(c0, d0, mul2(c1, d1)); }

// Four consecutive rows of one column.
struct __align__(16) V4 {
    f2 a, b;  // rows 0, 1 and 2, 3
};
static __device__ __forceinline__ V4 v4(f2 a, f2 b) {
    V4 r;
    r.a = a;
    r.b = b;
    return r;
}
static __device__ __forceinline__ V4 v4(const float4 &v) { return v4(pk(v.x, v.y), pk(v.z, v.w)); }
static __device__ __forceinline__ V4 zero4() { return v4(0ull, 0ull); }
static __device__ __forceinline__ V4 dup4(float v) { return v4(dup(v), dup(v)); }
static __device__ __forceinline__ V4 operator+(const V4 &x, const V4 &y) { return v4(add2(x.a, y.a), add2(x.b, y.b)); }
static __device__ __forceinline__ V4 operator-(const V4 &x, const V4 &y) { return v4(sub2(x.a, y.a), sub2(x.b, y.b)); }
static __device__ __forceinline__ V4 operator*(const V4 &x, const V4 &y) { return v4(mul2(x.a, y.a), mul2(x.b, y.b)); }
static __device__ __forceinline__ V4 fma4(const V4 &x, const V4 &y, const V4 &z) {
    return v4(fma2(x.a, y.a, z.a), fma2(x.b, y.b, z.b));
}
static __device__ __forceinline__ V4 dif4(const V4 &c0, const V4 &d0, const V4 &c1, const V4 &d1) {
    return fma4(c0, d0, c1 * d1);
}

// D- along z of the lane's four rows (cpu_modelling_kernels.cpp:201-258),
// neighbours by warp shuffles: c0 (f[z] - f[z-1]) + c1 (f[z+1] - f[z-2]).  The
// differences are scalar (their operands straddle the register pairs; packed
// ones would need a move per pair), the products packed.
static __device__ __forceinline__ V4 dminus_z(const V4 &c0, const V4 &c1, const V4 &f) {
    const float x = lo(f.a), y = hi(f.a), z = lo(f.b), w = hi(f.b);
    const float up_z = __shfl_up_sync(0xffffffffu, z, 1), up_w = __shfl_up_sync(0xffffffffu, w, 1);
    const float dn_x = __shfl_down_sync(0xffffffffu, x, 1);
    return v4(dif2(c0.a, pk(__fsub_rn(x, up_w), __fsub_rn(y, x)), c1.a, pk(__fsub_rn(y, up_z), __fsub_rn(z, up_w))),
              dif2(c0.b, pk(__fsub_rn(z, y), __fsub_rn(w, z)), c1.b, pk(__fsub_rn(w, x), __fsub_rn(dn_x, y))));
}
// D+ along z: c0 (f[z+1] - f[z]) + c1 (f[z+2] - f[z-1]).
static __device__ __forceinline__ V4 dplus_z(const V4 &c0, const V4 &c1, const V4 &f) {
    const float x = lo(f.a), y = hi(f.a), z = lo(f.b), w = hi(f.b);
    const float up_w = __shfl_up_sync(0xffffffffu, w, 1);
    const float dn_x = __shfl_down_sync(0xffffffffu, x, 1), dn_y = __shfl_down_sync(0xffffffffu, y, 1);
    return v4(dif2(c0.a, pk(__fsub_rn(y, x), __fsub_rn(z, y)), c1.a, pk(__fsub_rn(z, up_w), __fsub_rn(w, x))),
              dif2(c0.b, pk(__fsub_rn(w, z), __fsub_rn(dn_x, w)), c1.b, pk(__fsub_rn(dn_x, y), __fsub_rn(dn_y, z))));
}

}  // namespace s2d
