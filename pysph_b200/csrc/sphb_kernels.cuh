// sphb_kernels.cuh -- the smoothing kernels of the pair passes.
//
// Kern<KT> (KT = SPHB_KERNEL_*) gives, for one kernel type:
//   norm<DIM>()             _fac(1.0), the normalisation at h = 1
//   w_bf(q, fac)            W = fac val(q), branch-free (every piece
//                           computed, one selected): the tiled passes
//   gw_bf(q, ir, ih, fac_ih) dW/dr / r in the reference's sign convention,
//                           so grad_a W = (x_a - x_b) gw
//   w_in, gw_in<CLAMP>      the same for the list passes and their cell
//                           searches; without CLAMP inside the support only.
//                           gw_in keeps every factor of h outside the
//                           polynomial: with one h in the scene they are
//                           constants of the loop
// with fac = norm<DIM>() / h^DIM, ih = 1 / h, ir = 1 / r, fac_ih = fac ih,
// for T = float and double.  No form divides: the pair loops take one
// reciprocal square root per pair and, with one h in the scene, the dest's
// 1 / h.  For r = 0 they see a finite ir (inv_dist, dist_pair); every caller
// multiplies gw by r_ab = 0 there.

#pragma once

#include "sphb_common.cuh"

namespace sphb {

// Reciprocals and reciprocal square roots of the pair loops, without the
// branches and the denormal scaling of the general forms (no pair's
// denominators come near the denormals): a batch of pairs then is one
// straight run of instructions, which the compiler interleaves.  FP32: the
// hardware approximation.  FP64: the hardware's seed (relative error below
// 2^-19), then one third-order step from the binomial series of 1 / (1 - e)
// and 1 / sqrt(1 - e) in the seed's residual e.  Largest errors over 4 million
// mantissas, in units of the last place: 1 / x 0.51, r 0.75, 1 / r 0.99, r / h
// 0.50 (tests/test_pair_math_gpu.py has the bounds).
__device__ __forceinline__ float rcp_pair(float x)
{
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

__device__ __forceinline__ double rcp_pair(double x)
{
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-x, y, 1.0);
    return fma(y, fma(e, e, e), y);
}

__device__ __forceinline__ float rsqrt_pair(float x)
{
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// r and 1 / r from r^2, both from the one series: y (1 + p) and r^2 y (1 + p)
// with y the seed.  The rounding d of t = r^2 y enters each as d / 2, beside
// the last rounding.  Finite at r = 0, where r is 1e-100.
__device__ __forceinline__ double dist_pair(double r2, double &ir)
{
    const double x = fmax(r2, 1e-200);
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double t = x * y;
    const double e = fma(-t, y, 1.0);
    const double p = e * fma(0.375, e, 0.5);
    ir = fma(y, p, y);
    return fma(t, p, t);
}

// A product that no later sum contracts into an FMA.  The FP32C pair loops
// write every product and FMA out this way: a loop in which h is a constant
// and one in which it is the pair's then round alike, whatever the compiler
// would contract in each.
__device__ __forceinline__ float mul_pair(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_pair(double a, double b) { return __dmul_rn(a, b); }

// FP32: 1 / r from r^2; finite at r = 0, where r^2 times it is 0.
__device__ __forceinline__ float inv_dist(float r2) { return rsqrt_pair(fmaxf(r2, 1e-30f)); }

// q = r / h from r, h and 1 / h.  FP64: with the product's residual added back,
// so that q is rounded as a division rounds it.
__device__ __forceinline__ double over_h(double r, double h, double ih)
{
    const double q = r * ih;
    return fma(fma(-h, q, r), ih, q);
}

template <int KT>
struct Kern;

// CubicSplineKernel (S/base/kernels.pyx:349-454): support 2h,
// val = 1 - 1.5 q^2 (1 - q/2) (q <= 1), (2 - q)^3 / 4 (q <= 2), 0.
template <>
struct Kern<SPHB_KERNEL_CUBIC> {
    template <int DIM>
    __host__ __device__ static double norm() { return kfac_unit<DIM>(); }

    // q < 1: 1 + q^2 (0.75 q - 1.5); else t1^3 / 4 with t1 = max(2 - q, 0)
    template <typename T>
    __device__ __forceinline__ static T w_bf(T q, T fac)
    {
        const T t1 = fmax(T(2) - q, T(0));
        const T inner = fma(q * q, fma(T(0.75), q, T(-1.5)), T(1));
        const T outer = T(0.25) * (t1 * t1 * t1);
        return fac * (q < T(1) ? inner : outer);
    }

    // q < 1: (2.25 q - 3) ih; else -0.75 t1^2 / r
    template <typename T>
    __device__ __forceinline__ static T gw_bf(T q, T ir, T ih, T fac_ih)
    {
        const T t1 = fmax(T(2) - q, T(0));
        const T inner = (T(2.25) * q - T(3)) * ih;
        const T outer = T(-0.75) * t1 * t1 * ir;
        return fac_ih * (q < T(1) ? inner : outer);
    }

    template <bool CLAMP, typename T>
    __device__ __forceinline__ static T w_in(T q, T fac)
    {
        const T t1 = CLAMP ? fmax(T(2) - q, T(0)) : T(2) - q;
        const T inner = fma(q * q, fma(T(0.75), q, T(-1.5)), T(1));
        const T outer = T(0.25) * t1 * (t1 * t1);
        return fac * (q < T(1) ? inner : outer);
    }

    template <bool CLAMP, typename T>
    __device__ __forceinline__ static T gw_in(T q, T ir, T ih, T fac_ih)
    {
        const T t1 = CLAMP ? fmax(T(2) - q, T(0)) : T(2) - q;
        // (the polynomial's own constants stay exact: folding the factor into
        // them too would round each, and 2.25 q - 3 cancels)
        const T inner = fma(T(2.25), q, T(-3)) * (fac_ih * ih);
        const T outer = (T(-0.75) * fac_ih) * ir * (t1 * t1);
        return q < T(1) ? inner : outer;
    }
};

// QuinticSplineKernel (S/base/kernels.pyx:461-560), 2D: support 3h,
// fac = 7 / (478 pi).  Kept as the reference has them: W adds (1 - q)^5 with
// weight 1, and the gradient uses val = 5 t3^4 - 30 t2^4 + 75 t1^4 (the
// opposite sign of dW/dq), t_k = max(k - q, 0).
template <>
struct Kern<SPHB_KERNEL_QUINTIC> {
    template <int DIM>
    __host__ __device__ static double norm()
    {
        return DIM == 2 ? 7. / (478 * 3.141592653589793 * 1.0 * 1.0) : 0.0;
    }

    template <typename T>
    __device__ __forceinline__ static T p4(T t)
    {
        const T t2 = t * t;
        return t2 * t2;
    }

    template <typename T>
    __device__ __forceinline__ static T w_bf(T q, T fac)
    {
        const T t3 = fmax(T(3) - q, T(0));
        const T t2 = fmax(T(2) - q, T(0));
        const T t1 = fmax(T(1) - q, T(0));
        return fac * fma(p4(t1), t1, fma(T(-6) * p4(t2), t2, p4(t3) * t3));
    }

    template <typename T>
    __device__ __forceinline__ static T gw_bf(T q, T ir, T, T fac_ih)
    {
        const T t3 = fmax(T(3) - q, T(0));
        const T t2 = fmax(T(2) - q, T(0));
        const T t1 = fmax(T(1) - q, T(0));
        return fac_ih * ir * fma(T(75), p4(t1), fma(T(-30), p4(t2), T(5) * p4(t3)));
    }

    template <bool, typename T>
    __device__ __forceinline__ static T w_in(T q, T fac) { return w_bf(q, fac); }

    template <bool, typename T>
    __device__ __forceinline__ static T gw_in(T q, T ir, T ih, T fac_ih)
    {
        return gw_bf(q, ir, ih, fac_ih);
    }
};

// WendlandQuinticSplineKernel (S/base/kernels.pyx:562-640), 2D: support 2h,
// val = (1 - q/2)^4 (2q + 1).  Its _fac is written (7./4*PI*h*h), so the
// normalisation is 7 pi / 4 (not 7 / (4 pi)), kept as there.
template <>
struct Kern<SPHB_KERNEL_WENDLAND> {
    template <int DIM>
    __host__ __device__ static double norm()
    {
        return DIM == 2 ? (7. / 4 * 3.141592653589793 * 1.0 * 1.0) : 0.0;
    }

    template <typename T>
    __device__ __forceinline__ static T w_bf(T q, T fac)
    {
        const T t = fmax(fma(T(-0.5), q, T(1)), T(0));
        const T t2 = t * t;
        return fac * (t2 * t2 * fma(T(2), q, T(1)));
    }

    // dW/dr / r = -5 q t^3 fac / (h r) = -5 t^3 fac / h^2
    template <typename T>
    __device__ __forceinline__ static T gw_bf(T q, T, T ih, T fac_ih)
    {
        const T t = fmax(fma(T(-0.5), q, T(1)), T(0));
        return fac_ih * ih * (T(-5) * (t * t * t));
    }

    template <bool, typename T>
    __device__ __forceinline__ static T w_in(T q, T fac) { return w_bf(q, fac); }

    template <bool CLAMP, typename T>
    __device__ __forceinline__ static T gw_in(T q, T, T ih, T fac_ih)
    {
        T t = fma(T(-0.5), q, T(1));
        if (CLAMP) t = fmax(t, T(0));
        return (T(-5) * (fac_ih * ih)) * t * (t * t);
    }
};

}  // namespace sphb
