// trig.cuh -- branch-free sine/cosine for the bounded angles of the gauged
// stepper (link angles in (-pi, pi], plaquette angles in (-4pi, 4pi]).
//
// Method: additive (Cody-Waite) range reduction r = x - k*pi/2 with
// k = rint(x*2/pi) and pi/2 split into three parts, then the Taylor series of
// sin and cos about 0 evaluated by Horner's rule in r^2 on |r| <= pi/4, and
// the quadrant k mod 4 applied by selects.  FP64: terms through r^17 / r^16
// (truncation below 1e-17); FP32: through r^11 / r^10.  Valid for |x| up to
// about 2^20; tests/test_gpu_trig.py checks the result against CUDA's sin/cos.
// The FP64 step and the plane walkers take the batches further down, the FP32C
// pairs those of vec2.cuh: tests/test_gpu_trig_batch.py checks each against
// extended-precision values, tests/test_trig_polynomials.py the coefficients.
#pragma once
#include "common.cuh"

namespace scp {

template <class T>
struct TrigConsts;

template <>
struct TrigConsts<double> {
    // pi/2 = P1 + P2 + P3; P1 and P2 carry 33 significant bits each, so k*P1
    // and k*P2 are exact for |k| < 2^20; P3 is the rounded remainder.
    static constexpr double P1 = 0x1.921fb544p+0;
    static constexpr double P2 = 0x1.0b4611a6p-34;
    static constexpr double P3 = 0x1.3198a2e037073p-69;
    static constexpr double TWO_OVER_PI = 0x1.45f306dc9c883p-1;
};
template <>
struct TrigConsts<float> {
    // same split with 12-bit P1 and P2 (k*P exact for |k| < 2^12)
    static constexpr float P1 = 0x1.922p+0f;
    static constexpr float P2 = -0x1.2aep-18f;
    static constexpr float P3 = -0x1.de973ep-31f;
    static constexpr float TWO_OVER_PI = 0x1.45f306p-1f;
};

__device__ __forceinline__ double scp_rint(double x) { return rint(x); }
__device__ __forceinline__ float scp_rint(float x) { return rintf(x); }

// Taylor polynomials on |r| <= pi/4; s = r*r.
__device__ __forceinline__ void taylor_sc(double r, double *sn, double *cs) {
    const double s = r * r;
    // sin r = r (1 - s/3! + s^2/5! - ... + s^8/17!)
    double p = 2.8114572543455207632e-15;                  // 1/17!
    p = fma(p, s, -7.6471637318198164759e-13);             // -1/15!
    p = fma(p, s, 1.6059043836821614599e-10);              // 1/13!
    p = fma(p, s, -2.5052108385441718775e-8);              // -1/11!
    p = fma(p, s, 2.7557319223985890653e-6);               // 1/9!
    p = fma(p, s, -1.9841269841269841270e-4);              // -1/7!
    p = fma(p, s, 8.3333333333333333333e-3);               // 1/5!
    p = fma(p, s, -1.6666666666666666667e-1);              // -1/3!
    *sn = fma(r * s, p, r);
    // cos r = 1 - s/2! + s^2/4! - ... + s^8/16!
    double q = 4.7794773323873852974e-14;                  // 1/16!
    q = fma(q, s, -1.1470745597729724714e-11);             // -1/14!
    q = fma(q, s, 2.0876756987868098979e-9);               // 1/12!
    q = fma(q, s, -2.7557319223985890653e-7);              // -1/10!
    q = fma(q, s, 2.4801587301587301587e-5);               // 1/8!
    q = fma(q, s, -1.3888888888888888889e-3);              // -1/6!
    q = fma(q, s, 4.1666666666666666667e-2);               // 1/4!
    q = fma(q, s, -0.5);                                   // -1/2!
    *cs = fma(s, q, 1.0);
}
__device__ __forceinline__ void taylor_sc(float r, float *sn, float *cs) {
    const float s = r * r;
    float p = -2.5052108385441718775e-8f;                  // -1/11!
    p = fmaf(p, s, 2.7557319223985890653e-6f);             // 1/9!
    p = fmaf(p, s, -1.9841269841269841270e-4f);            // -1/7!
    p = fmaf(p, s, 8.3333333333333333333e-3f);             // 1/5!
    p = fmaf(p, s, -1.6666666666666666667e-1f);            // -1/3!
    *sn = fmaf(r * s, p, r);
    float q = -2.7557319223985890653e-7f;                  // -1/10!
    q = fmaf(q, s, 2.4801587301587301587e-5f);             // 1/8!
    q = fmaf(q, s, -1.3888888888888888889e-3f);            // -1/6!
    q = fmaf(q, s, 4.1666666666666666667e-2f);             // 1/4!
    q = fmaf(q, s, -0.5f);                                 // -1/2!
    *cs = fmaf(s, q, 1.0f);
}

// sin and cos of x, |x| <~ 2^20
template <class T>
__device__ __forceinline__ void sincos_bounded(T x, T *sn, T *cs) {
    using C = TrigConsts<T>;
    const T k = scp_rint(x * C::TWO_OVER_PI);
    T r = fma(-k, C::P1, x);
    r = fma(-k, C::P2, r);
    r = fma(-k, C::P3, r);
    T s, c;
    taylor_sc(r, &s, &c);
    const int q = ((int)k) & 3;
    // x = r + q*pi/2: rotate (s, c) by q quarter turns
    const T s1 = (q & 1) ? c : s;
    const T c1 = (q & 1) ? -s : c;
    *sn = (q & 2) ? -s1 : s1;
    *cs = (q & 2) ? -c1 : c1;
}

// sin and cos of any x: the bounded routine below 2^19, CUDA's sin / cos
// beyond (angles scaled by a user charge can be large)
__device__ __forceinline__ void sincos_any(double x, double *sn, double *cs) {
    if (fabs(x) < 0x1p19) {
        sincos_bounded(x, sn, cs);
    } else {
        *sn = sin(x);
        *cs = cos(x);
    }
}

// ---------------------------------------------------------------- batches
//
// Several angles of one site together (FP64), so that the range reduction --
// needed only beyond pi/4 (sine and cosine) or pi/2 (sine alone) -- is one
// branch for the batch: link and plaquette angles of a smooth state lie
// inside.  The reduced argument goes through near-minimax polynomials (Remez
// exchange on the absolute error, coefficients rounded to double):
//   |r| <= pi/4: sine to r^13 (8e-18), cosine to r^14 (2e-18)
//   |r| <= pi/2: sine to r^17 (4e-17, the rounding of 1/6)
// Two parts of pi (53 bits each) suffice for the reduction, since each product
// k * P is exact inside its fused multiply-add.

__device__ __forceinline__ unsigned abs_hi(double x) { return (unsigned)__double2hiint(x) & 0x7fffffffu; }
__device__ __forceinline__ double flip_sign(double x, unsigned bit) {   // bit: 0 or 1
    return __hiloint2double(__double2hiint(x) ^ (int)(bit << 31), __double2loint(x));
}
constexpr double kRintMagic = 6755399441055744.0;   // 1.5 * 2^52: adding it rounds to an integer

// sines and cosines of n angles, |a| < 2^20 (ANY: of any size, CUDA's sin and
// cos beyond 2^19, where the quadrant would leave the low word)
template <int n, bool ANY = false>
__device__ __forceinline__ void sincos_batch(const double (&ang)[n], double (&sn)[n], double (&cs)[n]) {
    double r[n];
    unsigned q[n], big = 0;
#pragma unroll
    for (int i = 0; i < n; i++) {
        r[i] = ang[i];
        q[i] = 0;
        big |= (abs_hi(ang[i]) >= 0x3fe921fbu) ? 1u : 0u;   // high word of pi/4
    }
    if (big) {
#pragma unroll
        for (int i = 0; i < n; i++) {
            const double t = __fma_rn(ang[i], 0x1.45f306dc9c883p-1, kRintMagic);   // 2/pi
            const double kq = __dadd_rn(t, -kRintMagic);
            r[i] = __fma_rn(-kq, 0x1.921fb54442d18p+0, ang[i]);
            r[i] = __fma_rn(-kq, 0x1.1a62633145c07p-54, r[i]);
            q[i] = (unsigned)__double2loint(t) & 3u;
        }
    }
#pragma unroll
    for (int i = 0; i < n; i++) {
        const double x = r[i], s = __dmul_rn(x, x);
        double p = __fma_rn(0x1.5d64c939ea033p-33, s, -0x1.ae5db478930bap-26);
        p = __fma_rn(p, s, 0x1.71de347564b0ep-19);
        p = __fma_rn(p, s, -0x1.a01a019ab4ae1p-13);
        p = __fma_rn(p, s, 0x1.111111110eb1fp-7);
        p = __fma_rn(p, s, -0x1.555555555553dp-3);
        sn[i] = __fma_rn(__dmul_rn(x, s), p, x);
        double c = __fma_rn(-0x1.8f806eafe7abbp-37, s, 0x1.1ee984acd9d7cp-29);
        c = __fma_rn(c, s, -0x1.27e4f7537ae12p-22);
        c = __fma_rn(c, s, 0x1.a01a019b6f8afp-16);
        c = __fma_rn(c, s, -0x1.6c16c16c13f18p-10);
        c = __fma_rn(c, s, 0x1.555555555553cp-5);
        c = __fma_rn(c, s, -0.5);
        cs[i] = __fma_rn(s, c, 1.0);
    }
    if (big) {   // x = r + q pi/2: rotate by q quarter turns
#pragma unroll
        for (int i = 0; i < n; i++) {
            const double s1 = (q[i] & 1) ? cs[i] : sn[i];
            const double c1 = (q[i] & 1) ? -sn[i] : cs[i];
            sn[i] = flip_sign(s1, q[i] >> 1);
            cs[i] = flip_sign(c1, q[i] >> 1);
            if (ANY && abs_hi(ang[i]) >= 0x41200000u) {   // 2^19
                sn[i] = sin(ang[i]);
                cs[i] = cos(ang[i]);
            }
        }
    }
}

// n angles replaced by their sines, |a| < 2^20
template <int n>
__device__ __forceinline__ void sin_batch(double (&x)[n]) {
    unsigned big = 0;
#pragma unroll
    for (int i = 0; i < n; i++) big |= (abs_hi(x[i]) >= 0x3ff921fbu) ? 1u : 0u;   // high word of pi/2
    if (big) {
#pragma unroll
        for (int i = 0; i < n; i++) {   // x = r + k pi: sin x = (-1)^k sin r
            const double t = __fma_rn(x[i], 0x1.45f306dc9c883p-2, kRintMagic);   // 1/pi
            const double kq = __dadd_rn(t, -kRintMagic);
            double r = __fma_rn(-kq, 0x1.921fb54442d18p+1, x[i]);
            r = __fma_rn(-kq, 0x1.1a62633145c07p-53, r);
            x[i] = flip_sign(r, (unsigned)__double2loint(t) & 1u);
        }
    }
#pragma unroll
    for (int i = 0; i < n; i++) {
        const double r = x[i], s = __dmul_rn(r, r);
        double p = __fma_rn(0x1.87c6cf61f7134p-49, s, -0x1.ae3f19d8db60ep-41);
        p = __fma_rn(p, s, 0x1.6123ba0dcfa88p-33);
        p = __fma_rn(p, s, -0x1.ae64547e9f285p-26);
        p = __fma_rn(p, s, 0x1.71de3a51c6a39p-19);
        p = __fma_rn(p, s, -0x1.a01a01a012737p-13);
        p = __fma_rn(p, s, 0x1.1111111111093p-7);
        p = __fma_rn(p, s, -0x1.5555555555555p-3);
        x[i] = __fma_rn(__dmul_rn(r, s), p, r);
    }
}

template <class T>
__device__ __forceinline__ T sin_bounded(T x) {
    T s, c;
    sincos_bounded(x, &s, &c);
    return s;
}

}  // namespace scp
