// The Skyrme mean field with the symmetry term at one node, for the fused
// path's kernels (k_fused.cu, k_smooth_fast.cu).
#pragma once

#include <cuda_runtime.h>

namespace hv {

// t^gamma to 1e-9 for t in [2^-8, 2^8] and |gamma| <= 8, in double: with t =
// 2^e m, m in [sqrt(1/2), sqrt(2)), log2 m is the series of 2 artanh(s) / ln 2
// in s = (m - 1) / (m + 1) (|s| < 0.172, left-out terms below 1e-10) and
// 2^(k + f) the Taylor series of e^(f ln 2) (|f| <= 1/2, below 3e-10).  27
// double operations without a table or a division; CUDA's pow, correct to an
// ulp over all of its range, has several times as many.
__device__ __forceinline__ double pow_mid(double t, double gamma) {
    const int hi = __double2hiint(t), e = (hi - 0x3fe6a09e) >> 20;
    const double m = __hiloint2double(hi - (e << 20), __double2loint(t)), den = m + 1.0;
    float rf;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(rf) : "f"((float)den));
    double r = (double)rf;
    r = r * (2.0 - den * r);
    const double s = (m - 1.0) * r, z = s * s;
    double p = 1.0 / 11.0;
    p = fma(p, z, 1.0 / 9.0);
    p = fma(p, z, 1.0 / 7.0);
    p = fma(p, z, 1.0 / 5.0);
    p = fma(p, z, 1.0 / 3.0);
    p = fma(p, z, 1.0);
    const double y = gamma * fma(s * 2.8853900817779268, p, (double)e);  // 2 / ln 2
    const double shift = 6755399441055744.0;                            // 1.5 * 2^52: rounds to an integer
    const double kd = y + shift;
    const double f = (y - (kd - shift)) * 0.69314718055994531;
    double q = 1.0 / 40320.0;
    q = fma(q, f, 1.0 / 5040.0);
    q = fma(q, f, 1.0 / 720.0);
    q = fma(q, f, 1.0 / 120.0);
    q = fma(q, f, 1.0 / 24.0);
    q = fma(q, f, 1.0 / 6.0);
    q = fma(q, f, 0.5);
    q = fma(q, f, 1.0);
    q = fma(q, f, 1.0);
    return __hiloint2double(__double2hiint(q) + (__double2loint(kd) << 20), __double2loint(q));
}

// t^gamma in float for t in [2^-20, 2^-8] and |gamma| <= 3 (gh + gl: gamma in two
// floats), to 2^-20.9 of it at gamma 7/6 and 2^-20.5 at 2: the logarithm's error
// (2^-22 of 1) times gamma ln 2, the exponential's 2^-22, two roundings.  The
// fast power rounds the product gamma log2 t at its own size, for another 2^-20.5
// where that passes 16.  Here the exponent's share gamma e goes into the result's
// exponent as an integer and an exact remainder, and only gamma log2 m, m in
// [sqrt(1/2), sqrt(2)), is rounded.
__device__ __forceinline__ float pow_low(float t, float gh, float gl) {
    const int hi = __float_as_int(t), e = (hi - 0x3f3504f3) >> 23;
    const float l = __log2f(__int_as_float(hi - (e << 23))), fe = (float)e, k = rintf(gh * fe);
    const float f = fmaf(gh, l, fmaf(gl, fe, fmaf(gh, fe, -k)));
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(f));
    return r * __int_as_float(((int)k + 127) << 23);
}

// Skyrme potential (include/physics.hpp:272-281, physics_formulas.hpp:70-77).
// A t and B t^gamma are some 300 MeV each and nearly cancel, so that a float
// power (CUDA's fast one: 3e-7 of its value) left more noise in the forces than
// the float storage of all fields together: 208Pb 64^3, rms error of a force
// component 3.2e-6 MeV/fm with __powf, 1.2e-6 with this form, and a third of
// the error in D(t) after 100 steps.  In float the sums are therefore formed in
// double and rounded once, where t >= 2^-8; below, B t^gamma is under 2 MeV and
// formed in float, in a nucleus's halo (down to 2^-20) with its exponent apart.
// The rest of the box, empty or holding the 2^-22 to 2^-32 that the FFT smoothing
// leaves, takes the fast power, whose share of U is small there.  208Pb 128^3,
// Skyrme kernel: 11.1 us with the fast power from 2^-8 down, 12.7 so, 14.8 with
// pow_low over the whole box, 12.1 with the doubles from 2^-20 on, which cost a
// step as much.  The double form (the fused FP64 path) keeps pow.
template <typename T>
__device__ __forceinline__ void skyrme_node(double A, double B, double C, double gamma, T rp, T rn, T &up, T &un) {
    if constexpr (sizeof(T) == 4) {
        const float inv_rho0 = 1.0f / 0.16f;
        const float tf = (rp + rn) * inv_rho0;
        if (tf >= 0.00390625f && tf < 255.0f && fabs(gamma) <= 8.0) {
            const double t = ((double)rp + (double)rn) * 6.25;
            const double base = A * t + B * pow_mid(t, gamma);
            const double iso = 12.5 * C * ((double)rn - (double)rp);
            up = (float)(base - iso);
            un = (float)(base + iso);
        } else {
            const float gh = (float)gamma;
            const float power = tf >= 9.5367432e-7f && tf < 0.00390625f && fabs(gamma) <= 3.0
                                    ? pow_low(tf, gh, (float)(gamma - (double)gh))
                                    : __powf(tf, gh);
            const float base = (float)A * tf + (float)B * power;
            const float iso = 2.0f * (float)C * ((rn - rp) * inv_rho0);
            up = base - iso;
            un = base + iso;
        }
    } else {
        const T t = (rp + rn) / T(0.16);
        const T base = A * t + B * pow(t, gamma);
        const T iso = T(2.0) * C * ((rn - rp) / T(0.16));
        up = base - iso;
        un = base + iso;
    }
}

}  // namespace hv
