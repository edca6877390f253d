// sphb_kernels.cuh -- the smoothing kernels of the pair passes.
//
// Kern<KT> (KT = SPHB_KERNEL_*) gives, for one kernel type:
//   norm<DIM>()             _fac(1.0), the normalisation at h = 1
//   w_bf(q, fac)            W = fac val(q), branch-free (every piece
//                           computed, one selected) for the list loops
//   gw_bf(q, ir, ih, fac_ih) dW/dr / r in the reference's sign convention,
//                           so grad_a W = (x_a - x_b) gw
// with fac = norm<DIM>() / h^DIM, ih = 1 / h, ir = 1 / r, fac_ih = fac ih,
// for T = float and double.  No form divides: the pair loops take one
// reciprocal square root per pair and, with one h in the scene, the dest's
// 1 / h.  For r = 0 they see a finite ir (inv_dist); every caller multiplies
// gw by r_ab = 0 there.

#pragma once

#include "sphb_common.cuh"

namespace sphb {

// 1 / r from r^2; finite at r = 0, where r^2 times it is 0.
__device__ __forceinline__ float inv_dist(float r2) { return rsqrtf(fmaxf(r2, 1e-30f)); }
__device__ __forceinline__ double inv_dist(double r2) { return rsqrt(fmax(r2, 1e-200)); }

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
};

}  // namespace sphb
