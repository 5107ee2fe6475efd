// vec2.cuh -- a pair of fp32 values computed with the sm_100 packed FP32
// instructions (__ffma2_rn, __fadd2_rn, __fmul2_rn): one instruction does the
// arithmetic of two lattice sites.
#pragma once
#include <cuda_runtime.h>

#include "trig.cuh"

namespace scp {

struct V2 {
    float2 v;
    __device__ __forceinline__ V2() {}
    __device__ __forceinline__ V2(float2 a) : v(a) {}
    __device__ __forceinline__ V2(float a, float b) { v.x = a; v.y = b; }
    __device__ __forceinline__ explicit V2(float s) { v.x = s; v.y = s; }
};

__device__ __forceinline__ V2 operator+(V2 a, V2 b) { return V2(__fadd2_rn(a.v, b.v)); }
__device__ __forceinline__ V2 operator*(V2 a, V2 b) { return V2(__fmul2_rn(a.v, b.v)); }
// a - b as b*(-1) + a: one rounding, like a scalar subtraction
__device__ __forceinline__ V2 operator-(V2 a, V2 b) { return V2(__ffma2_rn(b.v, make_float2(-1.f, -1.f), a.v)); }
__device__ __forceinline__ V2 operator-(V2 a) { return V2(-a.v.x, -a.v.y); }
__device__ __forceinline__ V2 fma2(V2 a, V2 b, V2 c) { return V2(__ffma2_rn(a.v, b.v, c.v)); }

// exact pair sums: s + e = a + b in each lane (Knuth two-sum)
__device__ __forceinline__ void two_sum2(V2 a, V2 b, V2 *s, V2 *e) {
    const V2 t = a + b;
    const V2 bb = t - a;
    *e = (a - (t - bb)) + (b - bb);
    *s = t;
}

// Batches of pairs of angles of one site pair, |x| <= 2^12: the reduction and
// Taylor polynomials of sincos_bounded<float> (trig.cuh) in packed arithmetic,
// with the range reduction -- needed only beyond pi/4, where the quadrant
// k = rint(x*2/pi) is not 0 -- as one branch for the batch.  The quadrant
// comes from adding 1.5*2^23, which leaves k in the low mantissa bits (round
// to nearest even, as rintf).
template <int n>
__device__ __forceinline__ bool any_beyond_quarter(const V2 (&x)[n]) {
    float m = 0.f;
    bool nan = false;
#pragma unroll
    for (int i = 0; i < n; i++) {
        m = fmaxf(m, fmaxf(fabsf(x[i].v.x), fabsf(x[i].v.y)));
        nan |= isnan(x[i].v.x) || isnan(x[i].v.y);
    }
    return m > 0.785398f || nan;
}
__device__ __forceinline__ V2 taylor_sin2(V2 r) {
    const V2 s = r * r;
    V2 p = fma2(V2(-2.5052108385441718775e-8f), s, V2(2.7557319223985890653e-6f));   // -1/11!, 1/9!
    p = fma2(p, s, V2(-1.9841269841269841270e-4f));                                   // -1/7!
    p = fma2(p, s, V2(8.3333333333333333333e-3f));                                    // 1/5!
    p = fma2(p, s, V2(-1.6666666666666666667e-1f));                                   // -1/3!
    return fma2(r * s, p, r);
}
__device__ __forceinline__ V2 taylor_cos2(V2 r) {
    const V2 s = r * r;
    V2 q = fma2(V2(-2.7557319223985890653e-7f), s, V2(2.4801587301587301587e-5f));   // -1/10!, 1/8!
    q = fma2(q, s, V2(-1.3888888888888888889e-3f));                                   // -1/6!
    q = fma2(q, s, V2(4.1666666666666666667e-2f));                                    // 1/4!
    q = fma2(q, s, V2(-0.5f));                                                         // -1/2!
    return fma2(s, q, V2(1.0f));
}

template <int n>
__device__ __forceinline__ void sincos2_batch(const V2 (&ang)[n], V2 (&sn)[n], V2 (&cs)[n]) {
    using C = TrigConsts<float>;
    const float MAGIC = 12582912.0f;   // 1.5 * 2^23
    V2 r[n];
    const bool big = any_beyond_quarter(ang);
#pragma unroll
    for (int i = 0; i < n; i++) r[i] = ang[i];
    if (big) {
#pragma unroll
        for (int i = 0; i < n; i++) {
            const V2 kq = fma2(ang[i], V2(C::TWO_OVER_PI), V2(MAGIC)) - V2(MAGIC);
            r[i] = fma2(kq, V2(-C::P1), ang[i]);
            r[i] = fma2(kq, V2(-C::P2), r[i]);
            r[i] = fma2(kq, V2(-C::P3), r[i]);
        }
    }
#pragma unroll
    for (int i = 0; i < n; i++) {
        sn[i] = taylor_sin2(r[i]);
        cs[i] = taylor_cos2(r[i]);
    }
    if (big) {   // x = r + k*pi/2: rotate (sin r, cos r) by k quarter turns, per lane
#pragma unroll
        for (int i = 0; i < n; i++) {
            const V2 t = fma2(ang[i], V2(C::TWO_OVER_PI), V2(MAGIC));
            const unsigned kx = __float_as_uint(t.v.x), ky = __float_as_uint(t.v.y);
            const unsigned gx = (kx & 2u) << 30, gy = (ky & 2u) << 30;   // sign flip for k = 2, 3 (mod 4)
            const float s1x = (kx & 1u) ? cs[i].v.x : sn[i].v.x, c1x = (kx & 1u) ? -sn[i].v.x : cs[i].v.x;
            const float s1y = (ky & 1u) ? cs[i].v.y : sn[i].v.y, c1y = (ky & 1u) ? -sn[i].v.y : cs[i].v.y;
            sn[i] = V2(__uint_as_float(__float_as_uint(s1x) ^ gx), __uint_as_float(__float_as_uint(s1y) ^ gy));
            cs[i] = V2(__uint_as_float(__float_as_uint(c1x) ^ gx), __uint_as_float(__float_as_uint(c1y) ^ gy));
        }
    }
}

// sines in place
template <int n>
__device__ __forceinline__ void sin2_batch(V2 (&x)[n]) {
    if (any_beyond_quarter(x)) {
        V2 s[n], c[n];
        sincos2_batch(x, s, c);
#pragma unroll
        for (int i = 0; i < n; i++) x[i] = s[i];
    } else {
#pragma unroll
        for (int i = 0; i < n; i++) x[i] = taylor_sin2(x[i]);
    }
}

}  // namespace scp
