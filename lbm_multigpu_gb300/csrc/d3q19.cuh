/*
 * d3q19.cuh -- per-cell D3Q19 operators of the stream-collide path (device code).
 *
 * Velocity ordering, moment basis and relaxation follow the reference
 * (LRTurbTest/LRMultiGPU7.cu, "LR7"):
 *   moments / basis          LR7:258-279
 *   mrt_collide (+ LES)      LR7:583-711
 *   *_Extrap rebuilds        LR7:713-897
 *   DynInlet3 MRT / BGK      MRTtest/DynInlet3.cu:599-832
 *   CPU_3D MRT               CPU_3D/CPU_3D.cpp:164-409
 * The arithmetic is organised for the GPU: populations are handled in
 * opposite-velocity pairs (even and odd parts), which halves the work of both
 * the forward moment transform and its inverse, and the Smagorinsky stress
 * |Pi_neq| is taken from the non-equilibrium moments the collision already has
 * instead of from 19 separately built equilibria (the two are the same linear
 * map: Pi_neq = sum c c f - rho/3 I - j j for every equilibrium used here).
 */
#pragma once

#include <cuda_runtime.h>

#include <cmath>
#include <stdint.h>

#include "lbm_kernels.cuh"

namespace lbm {

__host__ __device__ constexpr int cx(int q) {
    return (q == 1 || q == 5 || q == 8 || q == 10 || q == 15) ? 1 : (q == 3 || q == 6 || q == 7 || q == 12 || q == 17) ? -1 : 0;
}
__host__ __device__ constexpr int cy(int q) {
    return (q == 2 || q == 5 || q == 6 || q == 11 || q == 16) ? 1 : (q == 4 || q == 7 || q == 8 || q == 13 || q == 18) ? -1 : 0;
}
__host__ __device__ constexpr int cz(int q) { return (q >= 9 && q <= 13) ? 1 : (q >= 14) ? -1 : 0; }
__host__ __device__ constexpr int opp(int q) {
    return q == 0 ? 0 : q <= 4 ? ((q + 1) % 4 + 1) : q <= 8 ? ((q - 5 + 2) % 4 + 5) : q == 9 ? 14 : q == 14 ? 9 :
           q == 10 ? 17 : q == 17 ? 10 : q == 11 ? 18 : q == 18 ? 11 : q == 12 ? 15 : q == 15 ? 12 : q == 13 ? 16 : 13;
}
/* lattice weights (the equilibrium at rest), used for the offset storage f - w */
__host__ __device__ constexpr float wq(int q) {
    return q == 0 ? 1.f / 3.f : (q <= 4 || q == 9 || q == 14) ? 1.f / 18.f : 1.f / 36.f;
}

/* square root and reciprocal of the LES closure.  On the device in FP32 the
 * hardware approximations (a few ulp, far below the FP32 step-to-step
 * rounding the parity tolerance allows); in FP64 Newton's iteration from the
 * FP32 approximation, which takes 5 (square root) and 4 (reciprocal)
 * operations of the FP64 pipe.  That pipe does 2 operations per clock and SM
 * on this chip and bounds the FP64 kernels, so the seeds change format by
 * integer instructions (same exponent range, mantissa cut to 23 bits).
 * With the seed's relative error d, below 2^-21: the reciprocal's steps square
 * it (d^2, d^4); the square root's share one half-reciprocal of the seed's
 * precision, so that after the first, which leaves 1.5 d^2, the second gains
 * one more factor (1.5 d^3).  Both are far below 2^-53 then, which leaves the
 * rounding of the last operation: within an ulp of the IEEE result, and equal
 * to it but for near ties.  Arguments outside the FP32 range take the library
 * functions; IEEE operations on the host. */
#ifdef __CUDA_ARCH__
__device__ __forceinline__ bool fp32_range(double x) {
    /* 2^-100 <= x < 2^100, read from the exponent */
    return unsigned(__double2hiint(x)) - 0x39B00000u < 0x0C800000u;
}
__device__ __forceinline__ float fp32_cut(double x) {
    return __uint_as_float(((unsigned(__double2hiint(x)) - 0x38000000u) << 3) | (unsigned(__double2loint(x)) >> 29));
}
__device__ __forceinline__ double fp32_wide(float x) {
    const unsigned u = __float_as_uint(x);
    return __hiloint2double(int((u >> 3) + 0x38000000u), int(u << 29));
}
__device__ __forceinline__ double newton_sqrt(double x) {
    if (!fp32_range(x)) return sqrt(x);
    const float r = rsqrtf(fp32_cut(x));
    const double y = fp32_wide(r), h = fp32_wide(0.5f * r);
    double t = x * y;
    t = fma(fma(-t, t, x), h, t);
    return fma(fma(-t, t, x), h, t);
}
__device__ __forceinline__ double newton_rcp(double x) {
    if (!fp32_range(x)) return 1.0 / x;
    const double y = fp32_wide(__fdividef(1.0f, fp32_cut(x)));
    const double z = fma(fma(-x, y, 1.0), y, y);
    return fma(fma(-x, z, 1.0), z, z);
}
#endif
template <class T> __host__ __device__ __forceinline__ T lsqrt(T x) {
#ifdef __CUDA_ARCH__
    if constexpr (sizeof(T) == 4) return x > T(0) ? x * rsqrtf(x) : T(0);
    else return newton_sqrt(x);
#else
    return sqrt(x);
#endif
}
template <class T> __host__ __device__ __forceinline__ T lrcp(T x) {
#ifdef __CUDA_ARCH__
    if constexpr (sizeof(T) == 4) return __fdividef(1.0f, x);
    else return newton_rcp(x);
#else
    return T(1) / x;
#endif
}

/* Smagorinsky relaxation (LR7:683-685): tau = tau0/2 + sqrt(tau0^2 + 18 sqrt2 CS Q)/2.
 * The reference's CS enters where the textbook formula has Cs^2. */
template <class T> __host__ __device__ __forceinline__ T smag_omega(T omega, T cs, T qn) {
    T tau0 = lrcp(omega);
    T tau = T(0.5) * tau0 + T(0.5) * lsqrt(tau0 * tau0 + T(18) * cs * T(1.4142135623730951) * qn);
    return lrcp(tau);
}

/* Moment-space collision shared by the three MRT flavours.
 * VAR: MRT (LR7), MRT_DI3 (bgk_meq equilibria, then AddForce) or MRT_CPU3D
 * (CPU_3D's meq2 sign and rate-1 m13/m14). */
template <int VAR, class T>
__host__ __device__ __forceinline__ void collide_mrt(T f[19], T omega, bool les, T cs, T dpdy) {
    /* even / odd parts of the opposite pairs */
    const T sx = f[1] + f[3], dx = f[1] - f[3];
    const T sy = f[2] + f[4], dy = f[2] - f[4];
    const T sz = f[9] + f[14], dz = f[9] - f[14];
    const T a5 = f[5] + f[7], b5 = f[5] - f[7];
    const T a6 = f[6] + f[8], b6 = f[6] - f[8];
    const T a10 = f[10] + f[17], b10 = f[10] - f[17];
    const T a12 = f[12] + f[15], b12 = f[12] - f[15];
    const T a11 = f[11] + f[18], b11 = f[11] - f[18];
    const T a13 = f[13] + f[16], b13 = f[13] - f[16];

    const T axy = a5 + a6, axz = a10 + a12, ayz = a11 + a13;
    const T sax = sx + sy + sz, sdi = axy + axz + ayz;
    const T rho = f[0] + sax + sdi;
    const T Dx = b5 - b6 + b10 - b12, Dy = b5 + b6 + b11 - b13, Dz = b10 + b12 + b11 + b13;
    const T jx = dx + Dx, jy = dy + Dy, jz = dz + Dz;
    const T jxx = jx * jx, jyy = jy * jy, jzz = jz * jz;
    const T usq = jxx + jyy + jzz;

    /* non-equilibrium moments n_k = m_k - meq_k */
    T n1 = T(19) * ((sax + T(2) * sdi) - rho - usq);
    T n2 = T(12) * f[0] - T(4) * sax + sdi;
    T n9 = T(2) * sx - sy - sz + axy + axz - T(2) * ayz;
    T n10 = T(-4) * sx + T(2) * sy + T(2) * sz + axy + axz - T(2) * ayz;
    T n11 = sy - sz + axy - axz;
    T n12 = T(-2) * sy + T(2) * sz + axy - axz;
    const T m9eq = T(2) * jxx - (jyy + jzz), m11eq = jyy - jzz;
    if (VAR == MRT_DI3) {
        n2 -= T(3) * rho - T(5.5) * usq;
        n10 -= T(-0.5) * m9eq * T(0.333333333333);
        n12 -= T(-0.5) * m11eq;
    } else if (VAR == MRT_CPU3D) {
        n2 += T(7.53968254) * usq;
    } else {
        n2 -= T(7.53968254) * usq;
    }
    n9 -= m9eq;
    n11 -= m11eq;
    T n13 = (a5 - a6) - jx * jy;
    T n14 = (a11 - a13) - jy * jz;
    T n15 = (a10 - a12) - jx * jz;
    const T two3 = T(0.666666667);
    const T n4 = T(-4) * dx + Dx + two3 * jx;
    const T n6 = T(-4) * dy + Dy + two3 * jy;
    const T n8 = T(-4) * dz + Dz + two3 * jz;
    const T n16 = b5 - b6 - b10 + b12;
    const T n17 = -b5 - b6 + b11 - b13;
    const T n18 = b10 + b12 - b11 - b13;

    if (les) {
        /* Pi_neq from the stress moments: Pi_xx = n1/57 + n9/3,
         * Pi_yy + Pi_zz = n1/19 - Pi_xx, Pi_yy - Pi_zz = n11 */
        const T tr = n1 * T(1.0 / 19.0);
        const T pxx = n1 * T(1.0 / 57.0) + n9 * T(1.0 / 3.0);
        const T pyy = T(0.5) * (tr - pxx + n11), pzz = T(0.5) * (tr - pxx - n11);
        const T qn = lsqrt(pxx * pxx + pyy * pyy + pzz * pzz + T(2) * (n13 * n13 + n14 * n14 + n15 * n15));
        omega = smag_omega(omega, cs, qn);
    }
    /* relaxation: stress moments with omega, the rest to equilibrium */
    n9 *= omega;
    n11 *= omega;
    n15 *= omega;
    if (VAR == MRT_CPU3D) {
        /* CPU_3D relaxes m13 and m14 at rate 1 (CPU:246-248) */
    } else {
        n13 *= omega;
        n14 *= omega;
    }
    /* scaled by the row norms of the basis: f -= M^T diag(1/|M_k|^2) dm */
    const T g1 = n1 * T(1.0 / 2394.0), g2 = n2 * T(1.0 / 252.0);
    const T g4 = n4 * T(0.025), g6 = n6 * T(0.025), g8 = n8 * T(0.025);
    const T g9 = n9 * T(1.0 / 36.0), g10 = n10 * T(1.0 / 72.0);
    const T g11 = n11 * T(1.0 / 12.0), g12 = n12 * T(1.0 / 24.0);
    const T g13 = n13 * T(0.25), g14 = n14 * T(0.25), g15 = n15 * T(0.25);
    const T g16 = n16 * T(0.125), g17 = n17 * T(0.125), g18 = n18 * T(0.125);

    const T axis = T(-11) * g1 - T(4) * g2;
    const T diag = T(8) * g1 + g2;
    const T p9 = g9 - T(2) * g10;   /* -(9,10) combination on y/z axes */
    f[0] -= T(-30) * g1 + T(12) * g2;
    {   /* x axis pair (1,3) */
        const T e = axis + T(2) * g9 - T(4) * g10, o = T(-4) * g4;
        f[1] -= e + o;
        f[3] -= e - o;
    }
    {   /* y axis pair (2,4) */
        const T e = axis - p9 + g11 - T(2) * g12, o = T(-4) * g6;
        f[2] -= e + o;
        f[4] -= e - o;
    }
    {   /* z axis pair (9,14) */
        const T e = axis - p9 - g11 + T(2) * g12, o = T(-4) * g8;
        f[9] -= e + o;
        f[14] -= e - o;
    }
    const T dxy = diag + g9 + g10 + g11 + g12;
    const T dxz = diag + g9 + g10 - g11 - g12;
    const T dyz = diag - T(2) * g9 - T(2) * g10;
    {   /* (5,7): c = (1,1,0) */
        const T e = dxy + g13, o = g4 + g6 + g16 - g17;
        f[5] -= e + o;
        f[7] -= e - o;
    }
    {   /* (6,8): c = (-1,1,0) */
        const T e = dxy - g13, o = -g4 + g6 - g16 - g17;
        f[6] -= e + o;
        f[8] -= e - o;
    }
    {   /* (10,17): c = (1,0,1) */
        const T e = dxz + g15, o = g4 + g8 - g16 + g18;
        f[10] -= e + o;
        f[17] -= e - o;
    }
    {   /* (12,15): c = (-1,0,1) */
        const T e = dxz - g15, o = -g4 + g8 + g16 + g18;
        f[12] -= e + o;
        f[15] -= e - o;
    }
    {   /* (11,18): c = (0,1,1) */
        const T e = dyz + g14, o = g6 + g8 + g17 - g18;
        f[11] -= e + o;
        f[18] -= e - o;
    }
    {   /* (13,16): c = (0,-1,1) */
        const T e = dyz - g14, o = -g6 + g8 - g17 - g18;
        f[13] -= e + o;
        f[16] -= e - o;
    }
    if (VAR == MRT_DI3 && dpdy != T(0)) {
        /* AddForce (DI3:229-252) */
        const T a = T(0.0555555556) * T(3) * dpdy, b = T(0.0277777778) * T(3) * dpdy;
        f[2] -= a;
        f[4] += a;
        f[5] -= b;
        f[6] -= b;
        f[7] += b;
        f[8] += b;
        f[11] -= b;
        f[13] += b;
        f[16] -= b;
        f[18] += b;
    }
}

/* the square root of a non-negative x for the deviation collision: on the
 * device in FP32 x rsqrt(x + 1e-30), which is 0 at 0 without a branch */
template <class T> __host__ __device__ __forceinline__ T dsqrt(T x) {
#ifdef __CUDA_ARCH__
    if constexpr (sizeof(T) == 4) return x * rsqrtf(x + 1e-30f);
    else return newton_sqrt(x);
#else
    return sqrt(x);
#endif
}

/* the deviation collision's opposite-pair sums and final rebuild in packed
 * FP32 pairs (sm_100 and later: one instruction for two values) */
#ifndef LBM_DEV_F2
#define LBM_DEV_F2 1
#endif
#if defined(__CUDA_ARCH__) && __CUDA_ARCH__ >= 1000 && LBM_DEV_F2
#define LBM_F2_ON 1
#else
#define LBM_F2_ON 0
#endif
#if LBM_F2_ON
__device__ __forceinline__ float2 padd(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 pfma(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 psub(float2 a, float2 b) {
    unsigned long long ra = *reinterpret_cast<unsigned long long*>(&a);
    unsigned long long rb = *reinterpret_cast<unsigned long long*>(&b), rd;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(rd) : "l"(ra), "l"(rb));
    return *reinterpret_cast<float2*>(&rd);
}
#endif

/* LR7's MRT collision with Smagorinsky (LR7:583-711) in projected form, on
 * the deviations h = f - feq(1, (U, 0, 0)) of the populations from the
 * model's own equilibrium at density 1 and the reference velocity U along x
 * (the offsets of FP16 / BF16 storage), updated in place as such.
 *
 * The same map as collide_mrt<MRT>: there every non-conserved moment except
 * the five stresses m9, m11, m13, m14, m15 relaxes at rate 1, that is to its
 * equilibrium, so the post-collision moments are meq(rho, j) plus (1 - omega)
 * times the stress non-equilibrium, and the populations follow from them by
 * the inverse basis M^T diag(1 / |M_k|^2).  Only rho, j, the five stresses
 * and (for the eddy viscosity) m1 need the populations; even and odd parts
 * of each opposite pair are then rebuilt directly.  Subtracting the
 * equilibrium at (1, U) leaves the deviations: rho - 1, j - (U, 0, 0) in the
 * linear terms, j^2 - U^2 in the quadratic ones, meq(J) in the stresses.
 * Equilibrium moments (incompressible, rho0 = 1): meq1 = -11 rho + 19 j^2,
 * meq2 = 7.53968254 j^2 (LR7's sign), meq4,6,8 = -2/3 j, meq9 = 2 jx^2 -
 * jy^2 - jz^2, meq11 = jy^2 - jz^2, meq13,14,15 = jx jy, jy jz, jx jz,
 * meq10 = meq12 = meq16,17,18 = 0.
 * tau0 = 1 / omega and smag_k = 18 sqrt(2) CS are the Smagorinsky constants
 * (LR7:683-685), worked out once per launch.
 *
 * FP16 / BF16 storage and the learned closure (whose features are rounded to
 * BF16) turn a last-bit change of any operation here into a change of 16-bit
 * size, so the order of operations is part of these kernels' results; full
 * FP32 and FP64 populations take collide_mrt_pop. */
/* the moments of collide_mrt_dev that the populations give: density and
 * momentum deviations, j^2 - U^2, the stress equilibria and the
 * non-equilibrium stress moments n1, n9, n11, n13, n14, n15 */
template <class T> struct MrtDev {
    T rho, jx, jy, jz, q2, U2, m9eq, m11eq, jxy, jyz, jxz, n1, n9, n11, n13, n14, n15;
};

/* The projected collision is linear in the deviation from any equilibrium of
 * the model at rest, so it also takes full populations with U = 0 (the
 * rest equilibrium, alpha_q rho, then cancels exactly): collide_mrt_dev(f,
 * ..., 0) is collide_mrt<MRT> up to rounding. */
template <class T> __host__ __device__ __forceinline__ MrtDev<T> mrt_dev_moments(const T f[19], T U) {
#if LBM_F2_ON
    /* even and odd parts of the opposite pairs, two pairs per instruction */
    const float2 S1 = padd(make_float2(f[1], f[2]), make_float2(f[3], f[4]));
    const float2 D1 = psub(make_float2(f[1], f[2]), make_float2(f[3], f[4]));
    const float2 S2 = padd(make_float2(f[9], f[5]), make_float2(f[14], f[7]));
    const float2 D2 = psub(make_float2(f[9], f[5]), make_float2(f[14], f[7]));
    const float2 S3 = padd(make_float2(f[6], f[10]), make_float2(f[8], f[17]));
    const float2 D3 = psub(make_float2(f[6], f[10]), make_float2(f[8], f[17]));
    const float2 S4 = padd(make_float2(f[12], f[11]), make_float2(f[15], f[18]));
    const float2 D4 = psub(make_float2(f[12], f[11]), make_float2(f[15], f[18]));
    const T sx = S1.x, sy = S1.y, dx = D1.x, dy = D1.y, sz = S2.x, a5 = S2.y, dz = D2.x, b5 = D2.y;
    const T a6 = S3.x, a10 = S3.y, b6 = D3.x, b10 = D3.y, a12 = S4.x, a11 = S4.y, b12 = D4.x, b11 = D4.y;
#else
    const T sx = f[1] + f[3], dx = f[1] - f[3];
    const T sy = f[2] + f[4], dy = f[2] - f[4];
    const T sz = f[9] + f[14], dz = f[9] - f[14];
    const T a5 = f[5] + f[7], b5 = f[5] - f[7];
    const T a6 = f[6] + f[8], b6 = f[6] - f[8];
    const T a10 = f[10] + f[17], b10 = f[10] - f[17];
    const T a12 = f[12] + f[15], b12 = f[12] - f[15];
    const T a11 = f[11] + f[18], b11 = f[11] - f[18];
#endif
    const T a13 = f[13] + f[16], b13 = f[13] - f[16];
    const T axy = a5 + a6, axz = a10 + a12, ayz = a11 + a13;
    const T sdi = axy + axz + ayz;
    /* on deviations: rho - 1 and jx - U; on full populations (U = 0, the
     * model's equilibrium at rest then being the offset) rho and jx */
    const T rho = f[0] + (sx + sy + sz) + sdi;
    const T jx = dx + (b5 - b6) + (b10 - b12);
    const T jy = dy + (b5 + b6) + (b11 - b13);
    const T jz = dz + (b10 + b12) + (b11 + b13);
    const T Jx = jx + U;                                       /* the momentum */
    const T jxx = Jx * Jx, jyy = jy * jy, jzz = jz * jz;
    const T U2 = U * U;
    const T q2 = (jxx - U2) + (jyy + jzz);                     /* j^2 - U^2 */
    const T m9eq = T(2) * jxx - (jyy + jzz), m11eq = jyy - jzz;
    const T jxy = Jx * jy, jyz = jy * jz, jxz = Jx * jz;
    /* stress non-equilibrium moments (the linear parts of the deviations
     * plus those of the equilibrium at (1, U): 2 U^2 for m9, 0 else) */
    MrtDev<T> m;
    const T n9 = (T(2) * sx - sy - sz + axy + axz - T(2) * ayz) + (T(2) * U2 - m9eq);
    const T n11 = (sy - sz + axy - axz) - m11eq;
    const T n13 = (a5 - a6) - jxy, n14 = (a11 - a13) - jyz, n15 = (a10 - a12) - jxz;
    /* n1 = 19 (sdi - f0 - j^2) with the equilibrium's 19 U^2 */
    m.n1 = T(19) * ((sdi - f[0]) - q2);
    m.rho = rho, m.jx = jx, m.jy = jy, m.jz = jz, m.q2 = q2, m.U2 = U2, m.m9eq = m9eq, m.m11eq = m11eq;
    m.jxy = jxy, m.jyz = jyz, m.jxz = jxz, m.n9 = n9, m.n11 = n11, m.n13 = n13, m.n14 = n14, m.n15 = n15;
    return m;
}

/* the non-equilibrium stress Pi_neq (xx, yy, zz, xy, xz, yz) from the
 * moments, as collide_mrt forms it for the Smagorinsky model: Pi_xx =
 * n1/57 + n9/3, Pi_yy + Pi_zz = n1/19 - Pi_xx, Pi_yy - Pi_zz = n11 */
template <class T> __host__ __device__ __forceinline__ void mrt_dev_pi(const MrtDev<T>& m, T p[6]) {
    const T tr = m.n1 * T(1.0 / 19.0);
    p[0] = m.n1 * T(1.0 / 57.0) + m.n9 * T(1.0 / 3.0);
    p[1] = T(0.5) * (tr - p[0] + m.n11);
    p[2] = T(0.5) * (tr - p[0] - m.n11);
    p[3] = m.n13;
    p[4] = m.n15;
    p[5] = m.n14;
}

/* the Smagorinsky relaxation rate from the moments (LR7:683-685) */
template <class T> __host__ __device__ __forceinline__ T mrt_dev_les_omega(const MrtDev<T>& m, T tau0, T smag_k) {
    T p[6];
    mrt_dev_pi(m, p);
    const T qn = dsqrt(p[0] * p[0] + p[1] * p[1] + p[2] * p[2] + T(2) * (p[3] * p[3] + p[4] * p[4] + p[5] * p[5]));
    return lrcp(T(0.5) * tau0 + T(0.5) * dsqrt(tau0 * tau0 + smag_k * qn));
}

/* the products of the moments again from rho, j and the stresses, for a
 * caller that kept only those (fewer registers across a long wait) */
template <class T> __host__ __device__ __forceinline__ void mrt_dev_complete(MrtDev<T>& m, T U) {
    const T Jx = m.jx + U;
    const T jxx = Jx * Jx, jyy = m.jy * m.jy, jzz = m.jz * m.jz;
    m.U2 = U * U;
    m.q2 = (jxx - m.U2) + (jyy + jzz);
    m.m9eq = T(2) * jxx - (jyy + jzz), m.m11eq = jyy - jzz;
    m.jxy = Jx * m.jy, m.jyz = m.jy * m.jz, m.jxz = Jx * m.jz;
}

/* the post-collision deviations at the stress relaxation rate omega */
template <class T> __host__ __device__ __forceinline__ void mrt_dev_relax(T f[19], const MrtDev<T>& m, T omega) {
    const T rho = m.rho, jx = m.jx, jy = m.jy, jz = m.jz, q2 = m.q2, U2 = m.U2, m9eq = m.m9eq, m11eq = m.m11eq;
    const T jxy = m.jxy, jyz = m.jyz, jxz = m.jxz, n9 = m.n9, n11 = m.n11, n13 = m.n13, n14 = m.n14, n15 = m.n15;
    const T c1 = T(1) - omega;
    /* post-collision stresses less their value at (1, U), over the row norms */
    const T t9 = ((m9eq - T(2) * U2) + c1 * n9) * T(1.0 / 36.0);
    const T t11 = (m11eq + c1 * n11) * T(1.0 / 12.0);
    const T t13 = (jxy + c1 * n13) * T(0.25), t14 = (jyz + c1 * n14) * T(0.25), t15 = (jxz + c1 * n15) * T(0.25);
    /* rho / 19 + meq1 M1 / 2394 + meq2 M2 / 252 for the rest, axis and
     * diagonal rows (M1 = -30, -11, 8; M2 = 12, -4, 1) */
    const T A0 = T(1.0 / 19.0 + 330.0 / 2394.0) * rho + T(-570.0 / 2394.0 + 12.0 * 7.53968254 / 252.0) * q2;
    const T Aa = T(1.0 / 19.0 + 121.0 / 2394.0) * rho + T(-209.0 / 2394.0 - 4.0 * 7.53968254 / 252.0) * q2;
    const T Ad = T(1.0 / 19.0 - 88.0 / 2394.0) * rho + T(152.0 / 2394.0 + 7.53968254 / 252.0) * q2;
    /* odd parts: c.j / 6 on the axes, c.j / 12 on the diagonals */
    const T ox = jx * T(1.0 / 6.0), oy = jy * T(1.0 / 6.0), oz = jz * T(1.0 / 6.0);
    const T hx = jx * T(1.0 / 12.0), hy = jy * T(1.0 / 12.0), hz = jz * T(1.0 / 12.0);
    f[0] = A0;
    const T ayz9 = Aa - t9, d9 = Ad + t9;
    const T ex = Aa + T(2) * t9, ey = ayz9 + t11, ez = ayz9 - t11;
    const T bxy = d9 + t11, bxz = d9 - t11, byz = Ad - T(2) * t9;
    const T e5 = bxy + t13, e6 = bxy - t13, o5 = hx + hy, o6 = hy - hx;      /* xy: (5,7), (6,8) */
    const T e10 = bxz + t15, e12 = bxz - t15, o10 = hx + hz, o12 = hz - hx;  /* xz: (10,17), (12,15) */
    const T e11 = byz + t14, e13 = byz - t14, o11 = hy + hz, o13 = hz - hy;  /* yz: (11,18), (13,16) */
#if LBM_F2_ON
    {
        const float2 E = make_float2(ex, ey), O = make_float2(ox, oy);
        const float2 P = padd(E, O), M = psub(E, O);
        f[1] = P.x, f[2] = P.y, f[3] = M.x, f[4] = M.y;
    }
    f[9] = ez + oz;
    f[14] = ez - oz;
    {
        const float2 E = make_float2(e5, e6), O = make_float2(o5, o6);
        const float2 P = padd(E, O), M = psub(E, O);
        f[5] = P.x, f[6] = P.y, f[7] = M.x, f[8] = M.y;
    }
    {
        const float2 E = make_float2(e10, e12), O = make_float2(o10, o12);
        const float2 P = padd(E, O), M = psub(E, O);
        f[10] = P.x, f[12] = P.y, f[17] = M.x, f[15] = M.y;
    }
    {
        const float2 E = make_float2(e11, e13), O = make_float2(o11, o13);
        const float2 P = padd(E, O), M = psub(E, O);
        f[11] = P.x, f[13] = P.y, f[18] = M.x, f[16] = M.y;
    }
#else
    f[1] = ex + ox;
    f[3] = ex - ox;
    f[2] = ey + oy;
    f[4] = ey - oy;
    f[9] = ez + oz;
    f[14] = ez - oz;
    f[5] = e5 + o5;
    f[7] = e5 - o5;
    f[6] = e6 + o6;
    f[8] = e6 - o6;
    f[10] = e10 + o10;
    f[17] = e10 - o10;
    f[12] = e12 + o12;
    f[15] = e12 - o12;
    f[11] = e11 + o11;
    f[18] = e11 - o11;
    f[13] = e13 + o13;
    f[16] = e13 - o13;
#endif
}

template <class T>
__host__ __device__ __forceinline__ void collide_mrt_dev(T f[19], T omega, bool les, T tau0, T smag_k, T U) {
    const MrtDev<T> m = mrt_dev_moments(f, U);
    if (les) omega = mrt_dev_les_omega(m, tau0, smag_k);
    mrt_dev_relax(f, m, omega);
}

/* The same on populations, FP32 and FP64: the projected collision is linear in
 * the deviation from any equilibrium of the model at rest, so with U = 0 (the
 * rest equilibrium, alpha_q rho, then cancels exactly) it takes them as they
 * are.  About 60 operations for the moments, 25 for the eddy viscosity and 55
 * (FP32 73) for the rebuild, against some 325 in collide_mrt, which relaxes all
 * 19 moments: in FP64, where the operations are the bound, 1.05 M nodes took
 * 0.54 ms through collide_mrt and take 0.30 ms so.
 * Its moments: density, momentum, j^2, the stress equilibria, the
 * non-equilibrium stress moments and the trace tr = n1 / 19 of Pi_neq */
template <class T> struct MrtPop {
    T rho, jx, jy, jz, q2, m9eq, m11eq, jxy, jyz, jxz, tr, n9, n11, n13, n14, n15;
};

/* the linear parts alone (n9 .. tr without their equilibria) */
template <class T> __host__ __device__ __forceinline__ MrtPop<T> mrt_pop_sums(const T f[19]) {
    T sx, sy, sz, dx, dy, dz, a5, a6, a10, a11, a12, b5, b6, b10, b11, b12;
    /* even and odd parts of the opposite pairs; in FP32 on the device two
     * pairs per instruction */
#if LBM_F2_ON
    if constexpr (sizeof(T) == 4) {
        const float2 S1 = padd(make_float2(f[1], f[2]), make_float2(f[3], f[4]));
        const float2 D1 = psub(make_float2(f[1], f[2]), make_float2(f[3], f[4]));
        const float2 S2 = padd(make_float2(f[9], f[5]), make_float2(f[14], f[7]));
        const float2 D2 = psub(make_float2(f[9], f[5]), make_float2(f[14], f[7]));
        const float2 S3 = padd(make_float2(f[6], f[10]), make_float2(f[8], f[17]));
        const float2 D3 = psub(make_float2(f[6], f[10]), make_float2(f[8], f[17]));
        const float2 S4 = padd(make_float2(f[12], f[11]), make_float2(f[15], f[18]));
        const float2 D4 = psub(make_float2(f[12], f[11]), make_float2(f[15], f[18]));
        sx = S1.x, sy = S1.y, dx = D1.x, dy = D1.y, sz = S2.x, a5 = S2.y, dz = D2.x, b5 = D2.y;
        a6 = S3.x, a10 = S3.y, b6 = D3.x, b10 = D3.y, a12 = S4.x, a11 = S4.y, b12 = D4.x, b11 = D4.y;
    } else
#endif
    {
        sx = f[1] + f[3], dx = f[1] - f[3];
        sy = f[2] + f[4], dy = f[2] - f[4];
        sz = f[9] + f[14], dz = f[9] - f[14];
        a5 = f[5] + f[7], b5 = f[5] - f[7];
        a6 = f[6] + f[8], b6 = f[6] - f[8];
        a10 = f[10] + f[17], b10 = f[10] - f[17];
        a12 = f[12] + f[15], b12 = f[12] - f[15];
        a11 = f[11] + f[18], b11 = f[11] - f[18];
    }
    const T a13 = f[13] + f[16], b13 = f[13] - f[16];
    const T axy = a5 + a6, axz = a10 + a12, ayz = a11 + a13;
    const T ax = axy + axz, sdi = ax + ayz, syz = sy + sz;
    MrtPop<T> m;
    m.rho = f[0] + (sx + syz) + sdi;
    m.jx = dx + (b5 - b6) + (b10 - b12);
    m.jy = dy + (b5 + b6) + (b11 - b13);
    m.jz = dz + (b10 + b12) + (b11 + b13);
    m.n9 = (T(2) * sx - syz) + (ax - T(2) * ayz);
    m.n11 = (sy - sz) + (axy - axz);
    m.n13 = a5 - a6, m.n14 = a11 - a13, m.n15 = a10 - a12;
    m.tr = sdi - f[0];
    return m;
}

/* an inlet's or outlet's rebuild (extrap) of the moments' linear parts: every
 * moment kept but the momentum, set to (u_in, 0, 0) or (0, u_in, 0), or the
 * density, set to rho_bc.  A density change d is d / 19 in every population,
 * so m1 / 19 + 11 rho / 19 = sdi - f0 takes 11 d / 19 */
template <class T>
__host__ __device__ __forceinline__ void mrt_pop_extrap(MrtPop<T>& m, int type, T rho_bc, T u_in) {
    if (type == WEST_INLET || type == SOUTH_INLET) {
        m.jx = type == WEST_INLET ? u_in : T(0);
        m.jy = type == SOUTH_INLET ? u_in : T(0);
        m.jz = T(0);
    } else {
        const T d = rho_bc - m.rho;
        m.rho += d;
        m.tr += d * T(11.0 / 19.0);
    }
}

/* the products, and the non-equilibrium parts from the linear ones */
template <class T> __host__ __device__ __forceinline__ void mrt_pop_finish(MrtPop<T>& m) {
    const T jxx = m.jx * m.jx, jyy = m.jy * m.jy, yz = m.jz * m.jz + jyy;
    m.q2 = jxx + yz;
    m.m9eq = T(2) * jxx - yz;
    m.m11eq = jyy - m.jz * m.jz;
    m.jxy = m.jx * m.jy, m.jyz = m.jy * m.jz, m.jxz = m.jx * m.jz;
    m.n9 -= m.m9eq;
    m.n11 -= m.m11eq;
    m.n13 -= m.jxy, m.n14 -= m.jyz, m.n15 -= m.jxz;
    m.tr -= m.q2;
}

/* the Smagorinsky relaxation rate from the moments (LR7:683-685), with
 * Pi_yy^2 + Pi_zz^2 = ((Pi_yy + Pi_zz)^2 + (Pi_yy - Pi_zz)^2) / 2 */
template <class T> __host__ __device__ __forceinline__ T mrt_pop_les_omega(const MrtPop<T>& m, T tau0, T smag_k) {
    const T px = (m.tr + m.n9) * T(1.0 / 3.0), s = m.tr - px;
    const T off = m.n13 * m.n13 + m.n14 * m.n14 + m.n15 * m.n15;
    const T qn = dsqrt(px * px + T(0.5) * (s * s + m.n11 * m.n11) + T(2) * off);
    return lrcp(T(0.5) * tau0 + T(0.5) * dsqrt(tau0 * tau0 + smag_k * qn));
}

/* The constants of the rebuild: rho / 19 + meq1 M1 / 2394 + meq2 M2 / 252 for
 * the rest, axis and diagonal rows (M1 = -30, -11, 8; M2 = 12, -4, 1), a
 * share R of rho and Q of j^2 each, and the odd parts c.j WA on the axes, c.j WD
 * on the diagonals (j / 10 less 4 / 40, plus 1 / 40, of meq4 = -0.666666667 j
 * as LR7 writes it).  Mass and momentum come back exactly only if
 * R0 + 6 Ra + 12 Rd = 1, Q0 + 6 Qa + 12 Qd = 0 and 2 WA + 8 WD = 1 hold for the
 * rounded constants too; each rounded on its own they miss by 1e-8, which a
 * run in FP32 adds up step by step.  So the first of each sum is formed from
 * the others, which are such that it is representable: in FP32 1 / 63 is
 * rounded to a multiple of 2^-28 (R0 then is one of 2^-26), the others to
 * nearest. */
template <class T> struct PopRebuild {
    static constexpr T WD = T(0.1 - 0.025 * 0.666666667), WA = T(0.5 - 4.0 * double(WD));
    static constexpr T Rd = sizeof(T) == 4 ? T(4260880.0 / 268435456.0) : T(1.0 / 63.0), Ra = T(13.0 / 126.0);
    static constexpr T R0 = T(1.0 - 6.0 * double(Ra) - 12.0 * double(Rd));
    static constexpr T Qa = T(-209.0 / 2394.0 - 4.0 * 7.53968254 / 252.0), Qd = T(152.0 / 2394.0 + 7.53968254 / 252.0);
    static constexpr T Q0 = T(-6.0 * double(Qa) - 12.0 * double(Qd));
};
static_assert(2.0 * double(PopRebuild<float>::WA) + 8.0 * double(PopRebuild<float>::WD) == 1.0, "momentum");
static_assert(double(PopRebuild<float>::R0) + 6.0 * double(PopRebuild<float>::Ra) + 12.0 * double(PopRebuild<float>::Rd) == 1.0,
              "mass");
static_assert(double(PopRebuild<float>::Q0) + 6.0 * double(PopRebuild<float>::Qa) + 12.0 * double(PopRebuild<float>::Qd) == 0.0,
              "mass, quadratic part");

/* the post-collision populations at the stress relaxation rate omega.  In FP32
 * the density's share, by far the largest term, is added last, so that each
 * population is rounded once at its own size instead of three times
 * (statistics of a ragged channel against FP64, relative: 3.0e-7 so, 5.5e-7
 * with the density first, 3.1e-7 through collide_mrt; a uniform flow of 0.01 ..
 * 0.1 iterated 20,000 times loses less than 1e-7 of its mass, 1e-6 through
 * collide_mrt); FP64, whose 18 further operations would count, adds it first */
template <class T> __host__ __device__ __forceinline__ void mrt_pop_relax(T f[19], const MrtPop<T>& m, T omega) {
    constexpr bool LAST = sizeof(T) == 4;
    using K = PopRebuild<T>;
    const T rho = m.rho, jx = m.jx, jy = m.jy, jz = m.jz, q2 = m.q2;
    const T c1 = T(1) - omega;
    /* post-collision stresses over the row norms (the shear stresses still
     * times 4) */
    const T t9 = (m.m9eq + c1 * m.n9) * T(1.0 / 36.0);
    const T t11 = (m.m11eq + c1 * m.n11) * T(1.0 / 12.0);
    const T t13 = m.jxy + c1 * m.n13, t14 = m.jyz + c1 * m.n14, t15 = m.jxz + c1 * m.n15;
    const T Aa = LAST ? K::Qa * q2 : K::Ra * rho + K::Qa * q2, Ad = LAST ? K::Qd * q2 : K::Rd * rho + K::Qd * q2;
    constexpr T WA = K::WA, WD = K::WD, Q = T(0.25), Ra = K::Ra, Rd = K::Rd;
    f[0] = K::R0 * rho + K::Q0 * q2;
    const T ayz9 = Aa - t9, d9 = Ad + t9;
    const T ex = Aa + T(2) * t9, ey = ayz9 + t11, ez = ayz9 - t11;
    const T bxy = d9 + t11, bxz = d9 - t11, byz = Ad - T(2) * t9;
#if LBM_F2_ON
    if constexpr (sizeof(T) == 4) {
        const float2 wa = make_float2(WA, WA), na = make_float2(-WA, -WA), wd = make_float2(WD, WD),
                     nd = make_float2(-WD, -WD), qq = make_float2(Q, -Q), rr = make_float2(rho, rho),
                     ra = make_float2(Ra, Ra), rd = make_float2(Rd, Rd);
        /* E + O w and E - O w, with the density's share r rho */
        auto pair = [&](float2 E, float2 O, float2 w, float2 n, float2 r, T& p0, T& p1, T& m0, T& m1) {
            const float2 P = pfma(rr, r, pfma(O, w, E)), M = pfma(rr, r, pfma(O, n, E));
            p0 = P.x, p1 = P.y, m0 = M.x, m1 = M.y;
        };
        pair(make_float2(ex, ey), make_float2(jx, jy), wa, na, ra, f[1], f[2], f[3], f[4]);
        f[9] = ez + WA * jz + Ra * rho;
        f[14] = ez - WA * jz + Ra * rho;
        /* xy: (5,7), (6,8); xz: (10,17), (12,15); yz: (11,18), (13,16) */
        pair(pfma(make_float2(t13, t13), qq, make_float2(bxy, bxy)), make_float2(jx + jy, jy - jx), wd, nd, rd, f[5], f[6],
             f[7], f[8]);
        pair(pfma(make_float2(t15, t15), qq, make_float2(bxz, bxz)), make_float2(jx + jz, jz - jx), wd, nd, rd, f[10],
             f[12], f[17], f[15]);
        pair(pfma(make_float2(t14, t14), qq, make_float2(byz, byz)), make_float2(jy + jz, jz - jy), wd, nd, rd, f[11],
             f[13], f[18], f[16]);
        return;
    }
#endif
    f[1] = ex + WA * jx;
    f[3] = ex - WA * jx;
    f[2] = ey + WA * jy;
    f[4] = ey - WA * jy;
    f[9] = ez + WA * jz;
    f[14] = ez - WA * jz;
    const T e5 = bxy + Q * t13, e6 = bxy - Q * t13, o5 = jx + jy, o6 = jy - jx;
    f[5] = e5 + WD * o5;
    f[7] = e5 - WD * o5;
    f[6] = e6 + WD * o6;
    f[8] = e6 - WD * o6;
    const T e10 = bxz + Q * t15, e12 = bxz - Q * t15, o10 = jx + jz, o12 = jz - jx;
    f[10] = e10 + WD * o10;
    f[17] = e10 - WD * o10;
    f[12] = e12 + WD * o12;
    f[15] = e12 - WD * o12;
    const T e11 = byz + Q * t14, e13 = byz - Q * t14, o11 = jy + jz, o13 = jz - jy;
    f[11] = e11 + WD * o11;
    f[18] = e11 - WD * o11;
    f[13] = e13 + WD * o13;
    f[16] = e13 - WD * o13;
    if (LAST) {
#pragma unroll
        for (int q = 1; q < 19; ++q) f[q] += (q <= 4 || q == 9 || q == 14 ? Ra : Rd) * rho;
    }
}

/* type: an inlet or outlet whose neighbour's populations f are (mrt_pop_extrap
 * before the collision), or FLUID */
template <class T>
__host__ __device__ __forceinline__ void collide_mrt_pop(T f[19], T omega, bool les, T tau0, T smag_k, int type = FLUID,
                                                         T rho_bc = T(0), T u_in = T(0)) {
    MrtPop<T> m = mrt_pop_sums(f);
    if (type != FLUID) mrt_pop_extrap(m, type, rho_bc, u_in);
    mrt_pop_finish(m);
    if (les) omega = mrt_pop_les_omega(m, tau0, smag_k);
    mrt_pop_relax(f, m, omega);
}

/* BGK with the incompressible equilibrium w (rho + 3 c.j + 4.5 (c.j)^2 - 1.5 j^2)
 * (DI3:806-827, CPU:116-162), optional Smagorinsky and AddForce (DI3:830). */
template <class T> __host__ __device__ __forceinline__ void collide_bgk(T f[19], T omega, bool les, T cs, T dpdy) {
    T rho = 0, jx = 0, jy = 0, jz = 0;
#pragma unroll
    for (int q = 0; q < 19; ++q) {
        rho += f[q];
        if (cx(q)) jx += T(cx(q)) * f[q];
        if (cy(q)) jy += T(cy(q)) * f[q];
        if (cz(q)) jz += T(cz(q)) * f[q];
    }
    const T usq = jx * jx + jy * jy + jz * jz;
    if (les) {
        T pxx = 0, pyy = 0, pzz = 0, pxy = 0, pyz = 0, pxz = 0;
#pragma unroll
        for (int q = 1; q < 19; ++q) {
            if (cx(q)) pxx += f[q];
            if (cy(q)) pyy += f[q];
            if (cz(q)) pzz += f[q];
            if (cx(q) * cy(q)) pxy += T(cx(q) * cy(q)) * f[q];
            if (cy(q) * cz(q)) pyz += T(cy(q) * cz(q)) * f[q];
            if (cx(q) * cz(q)) pxz += T(cx(q) * cz(q)) * f[q];
        }
        const T third = rho * T(1.0 / 3.0);
        pxx -= third + jx * jx;
        pyy -= third + jy * jy;
        pzz -= third + jz * jz;
        pxy -= jx * jy;
        pyz -= jy * jz;
        pxz -= jx * jz;
        const T qn = lsqrt(pxx * pxx + pyy * pyy + pzz * pzz + T(2) * (pxy * pxy + pyz * pyz + pxz * pxz));
        omega = smag_omega(omega, cs, qn);
    }
    const T base = rho - T(1.5) * usq;
#pragma unroll
    for (int q = 0; q < 19; ++q) {
        const T cu = T(cx(q)) * jx + T(cy(q)) * jy + T(cz(q)) * jz;
        const T feq = T(wq(q)) * (base + T(3) * cu + T(4.5) * cu * cu);
        f[q] -= omega * (f[q] - feq);
    }
    if (dpdy != T(0)) {
        const T a = T(0.0555555556) * T(3) * dpdy, b = T(0.0277777778) * T(3) * dpdy;
        f[2] -= a;
        f[4] += a;
        f[5] -= b;
        f[6] -= b;
        f[7] += b;
        f[8] += b;
        f[11] -= b;
        f[13] += b;
        f[16] -= b;
        f[18] += b;
    }
}

/* density and non-equilibrium stress Pi_neq = sum c c f - rho/3 I - j j
 * (xx, yy, zz, xy, xz, yz) of the pulled populations: the input of the
 * learned subgrid closure (the quantity the Smagorinsky model takes the norm
 * of) */
template <class T> __host__ __device__ __forceinline__ void pi_neq(const T f[19], T& rho, T p[6]) {
    T r = 0, jx = 0, jy = 0, jz = 0, xx = 0, yy = 0, zz = 0, xy = 0, xz = 0, yz = 0;
#pragma unroll
    for (int q = 0; q < 19; ++q) {
        r += f[q];
        if (cx(q)) {
            jx += T(cx(q)) * f[q];
            xx += f[q];
        }
        if (cy(q)) {
            jy += T(cy(q)) * f[q];
            yy += f[q];
        }
        if (cz(q)) {
            jz += T(cz(q)) * f[q];
            zz += f[q];
        }
        if (cx(q) * cy(q)) xy += T(cx(q) * cy(q)) * f[q];
        if (cx(q) * cz(q)) xz += T(cx(q) * cz(q)) * f[q];
        if (cy(q) * cz(q)) yz += T(cy(q) * cz(q)) * f[q];
    }
    const T third = r * T(1.0 / 3.0);
    rho = r;
    p[0] = xx - third - jx * jx;
    p[1] = yy - third - jy * jy;
    p[2] = zz - third - jz * jz;
    p[3] = xy - jx * jy;
    p[4] = xz - jx * jz;
    p[5] = yz - jy * jz;
}

/* the models beside LR7's MRT */
template <class T>
__host__ __device__ __forceinline__ void collide_other(int model, T f[19], T omega, bool les, T cs, T dpdy) {
    switch (model) {
        case MRT_DI3: collide_mrt<MRT_DI3>(f, omega, les, cs, dpdy); break;
        case MRT_CPU3D: collide_mrt<MRT_CPU3D>(f, omega, les, cs, dpdy); break;
        default: collide_bgk(f, omega, les, cs, dpdy); break;
    }
}

template <class T>
__host__ __device__ __forceinline__ void collide(int model, T f[19], T omega, bool les, T cs, T dpdy) {
    if (model == MRT) collide_mrt<MRT>(f, omega, les, cs, dpdy);
    else collide_other(model, f, omega, les, cs, dpdy);
}

/* *_Extrap rebuild (LR7:713-897): keep every moment of the neighbour's
 * populations except density (outlets) or momentum (inlets); as a linear map
 *   f_q += (rho_new - rho)/19 + c_q.(j_new - j)/10 */
template <class T> __host__ __device__ __forceinline__ void extrap(int type, T f[19], T rho_bc, T u_in) {
    T rho = 0, jx = 0, jy = 0, jz = 0;
#pragma unroll
    for (int q = 0; q < 19; ++q) {
        rho += f[q];
        if (cx(q)) jx += T(cx(q)) * f[q];
        if (cy(q)) jy += T(cy(q)) * f[q];
        if (cz(q)) jz += T(cz(q)) * f[q];
    }
    T drho = 0, djx = 0, djy = 0, djz = 0;
    if (type == EAST_OUTLET || type == NORTH_OUTLET) {
        drho = rho_bc - rho;
    } else if (type == WEST_INLET) {
        djx = u_in - jx;
        djy = -jy;
        djz = -jz;
    } else if (type == SOUTH_INLET) {
        djx = -jx;
        djy = u_in - jy;
        djz = -jz;
    }
    const T r = drho * T(1.0 / 19.0);
    djx *= T(0.1);
    djy *= T(0.1);
    djz *= T(0.1);
#pragma unroll
    for (int q = 0; q < 19; ++q) f[q] += r + T(cx(q)) * djx + T(cy(q)) * djy + T(cz(q)) * djz;
}

/* ---- the alternate boundaries (node types DIR_WEST .. WEST_REG) ----
 * Per-cell restatements with the reference's own arithmetic and edge cases;
 * ny, nz are the domain's YDIM, ZDIM. */

/* the y/z edge copies shared by CPU_3D's DirichletWest and LR7's
 * xsymmetry_bot (CPU:417-470, LR7:901-945) */
template <class T> __host__ __device__ __forceinline__ void west_edges(T f[19], int y, int z, int ny, int nz) {
    if (y == 0 && z == 0) {
        f[2] = f[4], f[13] = f[18], f[11] = f[18], f[16] = f[18], f[6] = f[7], f[9] = f[14], f[12] = f[17];
    } else if (y == 0 && z == nz - 1) {
        f[4] = f[2], f[11] = f[13], f[18] = f[13], f[16] = f[13], f[6] = f[7], f[14] = f[9], f[17] = f[12];
    } else if (y == ny - 1 && z == 0) {
        f[4] = f[2], f[11] = f[16], f[18] = f[16], f[13] = f[16], f[7] = f[6], f[9] = f[14], f[12] = f[17];
    } else if (y == ny - 1 && z == nz - 1) {
        f[4] = f[2], f[16] = f[11], f[18] = f[11], f[13] = f[11], f[7] = f[6], f[14] = f[9], f[17] = f[12];
    } else {
        if (y == 0) f[2] = f[4], f[11] = f[13], f[16] = f[18], f[8] = f[5];
        else if (y == ny - 1) f[4] = f[2], f[13] = f[11], f[18] = f[16], f[5] = f[8];
    }
}

/* the corresponding copies at the east face (CPU:658-702, LR7:958-1006) */
template <class T> __host__ __device__ __forceinline__ void east_edges(T f[19], int y, int z, int ny, int nz) {
    if (y == 0 && z == 0) {
        f[2] = f[4], f[13] = f[18], f[11] = f[18], f[16] = f[18], f[5] = f[8], f[9] = f[14], f[10] = f[15];
    } else if (y == 0 && z == nz - 1) {
        f[2] = f[4], f[11] = f[13], f[18] = f[13], f[16] = f[13], f[5] = f[8], f[14] = f[9], f[15] = f[10];
    } else if (y == ny - 1 && z == 0) {
        f[4] = f[2], f[18] = f[16], f[11] = f[16], f[13] = f[16], f[8] = f[5], f[9] = f[14], f[10] = f[15];
    } else if (y == ny - 1 && z == nz - 1) {
        f[4] = f[2], f[13] = f[11], f[16] = f[11], f[18] = f[11], f[8] = f[5], f[14] = f[9], f[15] = f[10];
    } else {
        if (y == 0) f[2] = f[4], f[11] = f[13], f[16] = f[18], f[5] = f[8];
        else if (y == ny - 1) f[4] = f[2], f[13] = f[11], f[18] = f[16], f[8] = f[5];
    }
}

/* fused multiply-add as CPU_3D writes it (std::fma) */
template <class T> __host__ __device__ __forceinline__ T lfma(T a, T b, T c) {
#ifdef __CUDA_ARCH__
    return fma(a, b, c);
#else
    return std::fma(a, b, c);
#endif
}

/* DirichletWest (CPU:411-488): edges, then the unknowns from their
 * opposites with the inlet velocity u (v = w = 0), incompressible */
template <class T> __host__ __device__ __forceinline__ void dirichlet_west(T f[19], int y, int z, int ny, int nz, T u) {
    west_edges(f, y, z, ny, nz);
    if (!((y == 0 || y == ny - 1) && (z == 0 || z == nz - 1))) {
        if (z == 0) f[9] = f[14], f[10] = f[15], f[11] = f[16], f[13] = f[18];
        else if (z == nz - 1) f[14] = f[9], f[15] = f[10], f[16] = f[11], f[18] = f[13];
    }
    const T v = T(0), w = T(0);
    f[1] = lfma(T(0.0555555556), T(6) * u, f[3]);
    f[5] = lfma(T(0.0277777778), T(6) * (u + v), f[7]);
    f[8] = lfma(T(0.0277777778), T(6) * (u - v), f[6]);
    f[10] = lfma(T(0.0277777778), T(6) * (u + w), f[17]);
    f[15] = lfma(T(0.0277777778), T(6) * (u - w), f[12]);
}

/* the outlet velocity at rho = 1 from the known populations (CPU:649) */
template <class T> __host__ __device__ __forceinline__ T east_u(const T f[19]) {
    return -T(1) + (f[0] + f[2] + f[4] + f[9] + f[11] + f[13] + f[14] + f[16] + f[18] +
                    T(2) * (f[1] + f[8] + f[5] + f[10] + f[15]));
}

/* NeumannEast_Reg (CPU:570-650): edges (the corner copies of the east face,
 * the z-face copies without f12/f17), then the unknowns for rho = 1 */
template <class T> __host__ __device__ __forceinline__ void neumann_east(T f[19], int y, int z, int ny, int nz) {
    east_edges(f, y, z, ny, nz);
    if (!((y == 0 || y == ny - 1) && (z == 0 || z == nz - 1))) {
        if (z == 0) f[9] = f[14], f[10] = f[15], f[11] = f[16], f[13] = f[18];
        else if (z == nz - 1) f[14] = f[9], f[15] = f[10], f[16] = f[11], f[18] = f[13];
    }
    const T u = east_u(f), v = T(0), w = T(0);
    f[3] = f[1] - T(0.333333333) * u;
    f[7] = f[5] - T(0.166666667) * (u + v);
    f[6] = f[8] - T(0.166666667) * (u - v);
    f[17] = f[10] - T(0.166666667) * (u + w);
    f[12] = f[15] - T(0.166666667) * (u - w);
}

/* NeumannEast_Regularized (CPU:1056-1138) as written: rho = 1, u from the
 * known populations; the unknowns by non-equilibrium bounce-back where four
 * of the five read their own equilibrium twice (f3 = f1, f7 = f5,
 * f17 = f10, f12 = f15), then f = feq + Pi_neq projection */
template <class T> __host__ __device__ __forceinline__ void neumann_east_regularized(T f[19]) {
    const T rho = T(1), v = T(0), w = T(0);
    const T u = east_u(f);
    const T usq = u * u + v * v + w * w;
    T fe[19];
#pragma unroll
    for (int q = 0; q < 19; ++q) {
        const T cu = T(cx(q)) * u + T(cy(q)) * v + T(cz(q)) * w;
        const T wgt = q == 0 ? T(0.3333333333) : (q <= 4 || q == 9 || q == 14) ? T(0.0555555556) : T(0.0277777778);
        fe[q] = q == 0 ? wgt * (rho - T(1.5) * usq) : wgt * (rho + T(3) * cu + T(4.5) * cu * cu - T(1.5) * usq);
    }
    f[3] = fe[1] + f[1] - fe[1];
    f[7] = fe[5] + f[5] - fe[5];
    f[6] = fe[6] + f[8] - fe[8];
    f[17] = fe[10] + f[10] - fe[10];
    f[12] = fe[15] + f[15] - fe[15];
    T n[19];
#pragma unroll
    for (int q = 0; q < 19; ++q) n[q] = f[q] - fe[q];
    const T p11 = n[1] + n[3] + n[5] + n[6] + n[7] + n[8] + n[10] + n[12] + n[15] + n[17];
    const T p22 = n[2] + n[4] + n[5] + n[6] + n[7] + n[8] + n[11] + n[13] + n[16] + n[18];
    const T p33 = n[9] + n[14] + n[10] + n[12] + n[15] + n[17] + n[11] + n[13] + n[16] + n[18];
    const T p12 = n[5] + n[7] - n[6] - n[8];
    const T p13 = n[10] + n[17] - n[12] - n[15];
    const T p23 = n[11] + n[18] - n[13] - n[16];
    const T a = T(0.666666667), b = T(-0.333333333);
    f[0] = fe[0] + T(1.5) * (b * p11 + b * p22 + b * p33);
    f[1] = fe[1] + T(0.25) * (a * p11 + b * p22 + b * p33);
    f[2] = fe[2] + T(0.25) * (b * p11 + a * p22 + b * p33);
    f[3] = fe[3] + T(0.25) * (a * p11 + b * p22 + b * p33);
    f[4] = fe[4] + T(0.25) * (b * p11 + a * p22 + b * p33);
    f[5] = fe[5] + T(0.125) * (a * p11 + T(2) * p12 + a * p22 + b * p33);
    f[6] = fe[6] + T(0.125) * (a * p11 + T(2) * (-p12) + a * p22 + b * p33);
    f[7] = fe[7] + T(0.125) * (a * p11 + T(2) * p12 + a * p22 + b * p33);
    f[8] = fe[8] + T(0.125) * (a * p11 + T(2) * (-p12) + a * p22 + b * p33);
    f[9] = fe[9] + T(0.25) * (b * p11 + b * p22 + a * p33);
    f[10] = fe[10] + T(0.125) * (a * p11 + T(2) * p13 + b * p22 + a * p33);
    f[11] = fe[11] + T(0.125) * (b * p11 + T(2) * p23 + a * p22 + a * p33);
    f[12] = fe[12] + T(0.125) * (a * p11 + T(2) * (-p13) + b * p22 + a * p33);
    f[13] = fe[13] + T(0.125) * (b * p11 + T(2) * (-p23) + a * p22 + a * p33);
    f[14] = fe[14] + T(0.25) * (b * p11 + b * p22 + a * p33);
    f[15] = fe[15] + T(0.125) * (a * p11 + T(2) * (-p13) + b * p22 + a * p33);
    f[16] = fe[16] + T(0.125) * (b * p11 + T(2) * (-p23) + a * p22 + a * p33);
    f[17] = fe[17] + T(0.125) * (a * p11 + T(2) * p13 + b * p22 + a * p33);
    f[18] = fe[18] + T(0.125) * (b * p11 + T(2) * p23 + a * p22 + a * p33);
}

/* xsymmetry_bot / xsymmetry_top (LR7:899-1016): specular planes at x = 0
 * and x = nx - 1 with their y/z edge copies */
template <class T> __host__ __device__ __forceinline__ void xsym_bot(T f[19], int y, int z, int ny, int nz) {
    west_edges(f, y, z, ny, nz);
    f[1] = f[3], f[5] = f[6], f[8] = f[7], f[10] = f[12], f[15] = f[17];
}
template <class T> __host__ __device__ __forceinline__ void xsym_top(T f[19], int y, int z, int ny, int nz) {
    east_edges(f, y, z, ny, nz);
    f[3] = f[1], f[6] = f[5], f[7] = f[8], f[12] = f[10], f[17] = f[15];
}

/* ysymmetry_top / _bot (CPU:861-916), zsymmetry_top / _bot (CPU:917-972) */
template <class T> __host__ __device__ __forceinline__ void ysym(T f[19], bool top, int z, int nz) {
    if (z == 0) f[9] = f[14], f[10] = f[15], f[11] = f[16], f[12] = f[17], f[13] = f[18];
    if (z == nz - 1) f[14] = f[9], f[15] = f[10], f[16] = f[11], f[17] = f[12], f[18] = f[13];
    if (top) f[4] = f[2], f[7] = f[6], f[8] = f[5], f[13] = f[11], f[18] = f[16];
    else f[2] = f[4], f[6] = f[7], f[5] = f[8], f[11] = f[13], f[16] = f[18];
}
template <class T> __host__ __device__ __forceinline__ void zsym(T f[19], bool top, int y, int ny) {
    if (y == 0) f[2] = f[4], f[6] = f[7], f[5] = f[8], f[11] = f[13], f[16] = f[18];
    if (y == ny - 1) f[4] = f[2], f[7] = f[6], f[8] = f[5], f[13] = f[11], f[18] = f[16];
    if (top) f[14] = f[9], f[15] = f[10], f[16] = f[11], f[17] = f[12], f[18] = f[13];
    else f[9] = f[14], f[10] = f[15], f[11] = f[16], f[12] = f[17], f[13] = f[18];
}

/* West_Reg (BC1/LRMultiGPU7.cu:789-870): the node's own populations keep
 * rho and every non-momentum moment, the momentum becomes (u, 0, w) with
 * w = 0.01 at t = 1000, 2000, 3000 (the reference's perturbation).  The
 * reference rebuilds the node from all 19 MRT moments; with only the
 * momentum rows changed that is f += c . (j_target - j) / 10 (the momentum
 * columns of the inverse transform are c / 10), same in real arithmetic,
 * FP32 results within rounding of the reference's */
template <class T> __host__ __device__ __forceinline__ void west_reg(T f[19], T u, int t) {
    const T w = (t == 1000 || t == 2000 || t == 3000) ? T(0.01) : T(0);
    T jx = 0, jy = 0, jz = 0;
#pragma unroll
    for (int q = 0; q < 19; ++q) {
        if (cx(q)) jx += T(cx(q)) * f[q];
        if (cy(q)) jy += T(cy(q)) * f[q];
        if (cz(q)) jz += T(cz(q)) * f[q];
    }
    const T dx = T(0.1) * (u - jx), dy = T(0.1) * (T(0) - jy), dz = T(0.1) * (w - jz);
#pragma unroll
    for (int q = 0; q < 19; ++q) f[q] += T(cx(q)) * dx + T(cy(q)) * dy + T(cz(q)) * dz;
}

/* DirichletWest_Reg (CPU:379-453): x = 0 with velocity (0, v, 0), its y
 * edge copies, then the z face copies; DirichletNorth_Reg / _South_Reg
 * (CPU:578-745): y = ny - 1 / y = 0 walls moving with (u, 0, 0) after the
 * z face copies.  Unknowns from their opposites plus 6 w_q c_q . u (rho = 1) */
template <class T> __host__ __device__ __forceinline__ void z_face_copies(T f[19], int z, int nz) {
    if (z == 0) f[9] = f[14], f[10] = f[15], f[11] = f[16], f[12] = f[17], f[13] = f[18];
    else if (z == nz - 1) f[14] = f[9], f[15] = f[10], f[16] = f[11], f[17] = f[12], f[18] = f[13];
}
template <class T> __host__ __device__ __forceinline__ void dirichlet_west_v(T f[19], int y, int z, int ny, int nz, T v) {
    if (y == 0) f[2] = f[4], f[6] = f[7], f[11] = f[13], f[16] = f[18];
    else if (y == ny - 1) f[4] = f[2], f[7] = f[6], f[13] = f[11], f[18] = f[16];
    z_face_copies(f, z, nz);
    const T u = T(0), w = T(0);
    f[1] = f[3] + T(0.33333333) * u;
    f[5] = f[7] + T(0.166666667) * (u + v);
    f[8] = f[6] + T(0.166666667) * (u - v);
    f[10] = f[17] + T(0.166666667) * (u + w);
    f[15] = f[12] + T(0.166666667) * (u - w);
}
template <class T> __host__ __device__ __forceinline__ void dirichlet_north(T f[19], int z, int nz, T u) {
    z_face_copies(f, z, nz);
    const T v = T(0), w = T(0);
    f[4] = f[2] - T(0.33333333) * v;
    f[7] = f[5] - T(0.166666667) * (u + v);
    f[8] = f[6] + T(0.166666667) * (u - v);
    f[13] = f[16] - T(0.166666667) * (v - w);
    f[18] = f[11] - T(0.166666667) * (v + w);
}
template <class T> __host__ __device__ __forceinline__ void dirichlet_south(T f[19], int z, int nz, T u) {
    z_face_copies(f, z, nz);
    const T v = T(0), w = T(0);
    f[2] = f[4] + T(0.33333333) * v;
    f[5] = f[7] + T(0.166666667) * (u + v);
    f[6] = f[8] - T(0.166666667) * (u - v);
    f[16] = f[13] + T(0.166666667) * (v - w);
    f[11] = f[18] + T(0.166666667) * (v + w);
}

/* the dispatch for a node of an alternate-boundary type */
template <class T>
__host__ __device__ __forceinline__ void alt_boundary(int type, T f[19], int x, int y, int z, int nx, int ny, int nz,
                                                      T u_in, int t) {
    (void)x, (void)nx;
    switch (type) {
        case DIR_WEST: dirichlet_west(f, y, z, ny, nz, u_in); break;
        case NEU_EAST: neumann_east(f, y, z, ny, nz); break;
        case NEU_EAST_REG: neumann_east_regularized(f); break;
        case XSYM_TOP: xsym_top(f, y, z, ny, nz); break;
        case XSYM_BOT: xsym_bot(f, y, z, ny, nz); break;
        case YSYM_TOP: ysym(f, true, z, nz); break;
        case YSYM_BOT: ysym(f, false, z, nz); break;
        case ZSYM_TOP: zsym(f, true, y, ny); break;
        case ZSYM_BOT: zsym(f, false, y, ny); break;
        case WEST_REG: west_reg(f, u_in, t); break;
        case DIR_WEST_V: dirichlet_west_v(f, y, z, ny, nz, u_in); break;
        case DIR_NORTH: dirichlet_north(f, z, nz, u_in); break;
        case DIR_SOUTH: dirichlet_south(f, z, nz, u_in); break;
        default: break;
    }
}

/* Regularised velocity boundary for a moving lid on any face (the reference's
 * DirichletWest_Regularized, CPU:974-1054, written per face): density from the
 * known populations, unknowns by non-equilibrium bounce-back, then
 * f = feq + 4.5 w_q (c_q c_q - I/3) : Pi_neq. */
template <class T>
__host__ __device__ __forceinline__ void lid(T f[19], int face, T ux, T uy, T uz, bool quirk = false) {
    const int axis = face >> 1;
    const int sgn = (face & 1) ? -1 : 1;
    T s0 = 0, s1 = 0;
#pragma unroll
    for (int q = 0; q < 19; ++q) {
        const int cn = (axis == 0 ? cx(q) : axis == 1 ? cy(q) : cz(q)) * sgn;
        if (cn == 0) s0 += f[q];
        else if (cn < 0) s1 += f[q];
    }
    const T un = (axis == 0 ? ux : axis == 1 ? uy : uz) * T(sgn);
    const T rho = un + (s0 + T(2) * s1);
    const T usq = ux * ux + uy * uy + uz * uz;
    T feq[19];
#pragma unroll
    for (int q = 0; q < 19; ++q) {
        const T cu = T(cx(q)) * ux + T(cy(q)) * uy + T(cz(q)) * uz;
        feq[q] = T(wq(q)) * (rho + T(3) * cu + T(4.5) * cu * cu - T(1.5) * usq);
    }
    if (quirk) {
        /* CPU_3D writes (v+w)*(u+w) and (-v+w)*(u+w) for the squares of
         * populations 11 and 13 (CPU:1012, 1014) */
        feq[11] = T(wq(11)) * (rho + T(3) * (uy + uz) + T(4.5) * (uy + uz) * (ux + uz) - T(1.5) * usq);
        feq[13] = T(wq(13)) * (rho + T(3) * (-uy + uz) + T(4.5) * (-uy + uz) * (ux + uz) - T(1.5) * usq);
    }
    T g[19];
#pragma unroll
    for (int q = 0; q < 19; ++q) g[q] = f[q] - feq[q];
#pragma unroll
    for (int q = 0; q < 19; ++q) {
        const int cn = (axis == 0 ? cx(q) : axis == 1 ? cy(q) : cz(q)) * sgn;
        if (cn > 0) g[q] = g[opp(q)];
    }
    if (quirk && face == 0) {
        /* CPU:1023 sets f8 = feq6 + f6 - feq6 */
        g[8] = (feq[6] + f[6] - feq[6]) - feq[8];
    }
    T P[6] = {0, 0, 0, 0, 0, 0};
#pragma unroll
    for (int q = 1; q < 19; ++q) {
        P[0] += T(cx(q) * cx(q)) * g[q];
        P[1] += T(cy(q) * cy(q)) * g[q];
        P[2] += T(cz(q) * cz(q)) * g[q];
        P[3] += T(cx(q) * cy(q)) * g[q];
        P[4] += T(cy(q) * cz(q)) * g[q];
        P[5] += T(cx(q) * cz(q)) * g[q];
    }
    const T tr = (P[0] + P[1] + P[2]) * T(1.0 / 3.0);
#pragma unroll
    for (int q = 0; q < 19; ++q) {
        const T s = T(cx(q) * cx(q)) * P[0] + T(cy(q) * cy(q)) * P[1] + T(cz(q) * cz(q)) * P[2] +
                    T(2 * cx(q) * cy(q)) * P[3] + T(2 * cy(q) * cz(q)) * P[4] + T(2 * cx(q) * cz(q)) * P[5] - tr;
        f[q] = feq[q] + T(wq(q)) * T(4.5) * s;
    }
}

/* PhysicalMoments (LR7:380-391): rho, j, m9, m11, m13, m14, m15 */
template <class T> __host__ __device__ __forceinline__ void physical_moments(const T f[19], T mom[9]) {
    const T sx = f[1] + f[3], sy = f[2] + f[4], sz = f[9] + f[14];
    const T a5 = f[5] + f[7], a6 = f[6] + f[8], a10 = f[10] + f[17], a12 = f[12] + f[15];
    const T a11 = f[11] + f[18], a13 = f[13] + f[16];
    const T b5 = f[5] - f[7], b6 = f[6] - f[8], b10 = f[10] - f[17], b12 = f[12] - f[15];
    const T b11 = f[11] - f[18], b13 = f[13] - f[16];
    const T axy = a5 + a6, axz = a10 + a12, ayz = a11 + a13;
    mom[0] = f[0] + sx + sy + sz + axy + axz + ayz;
    mom[1] = (f[1] - f[3]) + b5 - b6 + b10 - b12;
    mom[2] = (f[2] - f[4]) + b5 + b6 + b11 - b13;
    mom[3] = (f[9] - f[14]) + b10 + b12 + b11 + b13;
    mom[4] = T(2) * sx - sy - sz + axy + axz - T(2) * ayz;
    mom[5] = sy - sz + axy - axz;
    mom[6] = a5 - a6;
    mom[7] = a11 - a13;
    mom[8] = a10 - a12;
}

/* StrainRate (LR7:351-377) with the reference's omega = 1, m1 = 0, dx = 1 */
template <class T> __host__ __device__ __forceinline__ void strain_rate(const T mom[9], T S[6]) {
    const T u = mom[1], v = mom[2], w = mom[3];
    const T n9 = mom[4] - (T(2) * u * u - (v * v + w * w));
    const T n11 = mom[5] - (v * v - w * w);
    S[0] = T(-0.5) * n9;
    S[1] = T(0.25) * (n9 - T(3) * n11);
    S[2] = T(0.25) * (n9 + T(3) * n11);
    S[3] = T(-1.5) * (mom[6] - u * v);
    S[4] = T(-1.5) * (mom[7] - v * w);
    S[5] = T(-1.5) * (mom[8] - u * w);
}

template <class T> __host__ __device__ __forceinline__ T strain_mag(const T S[6]) {
    return sqrt(T(2) * (S[0] * S[0] + S[1] * S[1] + S[2] * S[2] + T(2) * (S[3] * S[3] + S[4] * S[4] + S[5] * S[5])));
}

/* equilibrium moments with the non-equilibrium stress scaled by SF, back to
 * populations (InvertPhysicalMoments, LR7:421-465) */
template <class T> __host__ __device__ __forceinline__ void invert_scaled(const T mom[9], T SF, T f[19]) {
    const T rho = mom[0], u = mom[1], v = mom[2], w = mom[3];
    const T usq = u * u + v * v + w * w;
    const T one = T(1) - SF;
    const T m1 = T(-11) * rho + T(19) * usq, m2 = T(7.53968254) * usq;
    const T m4 = T(-0.666666667) * u, m6 = T(-0.666666667) * v, m8 = T(-0.666666667) * w;
    const T m9 = mom[4] * SF + one * (T(2) * u * u - (v * v + w * w));
    const T m11 = mom[5] * SF + one * (v * v - w * w);
    const T m13 = mom[6] * SF + one * u * v;
    const T m14 = mom[7] * SF + one * v * w;
    const T m15 = mom[8] * SF + one * u * w;
    const T g0 = rho * T(1.0 / 19.0), g1 = m1 * T(1.0 / 2394.0), g2 = m2 * T(1.0 / 252.0);
    const T gu = u * T(0.1), gv = v * T(0.1), gw = w * T(0.1);
    const T g4 = m4 * T(0.025), g6 = m6 * T(0.025), g8 = m8 * T(0.025);
    const T g9 = m9 * T(1.0 / 36.0), g11 = m11 * T(1.0 / 12.0);
    const T g13 = m13 * T(0.25), g14 = m14 * T(0.25), g15 = m15 * T(0.25);
    const T axis = g0 + T(-11) * g1 - T(4) * g2;
    const T diag = g0 + T(8) * g1 + g2;
    f[0] = g0 + T(-30) * g1 + T(12) * g2;
    f[1] = axis + T(2) * g9 + (gu - T(4) * g4);
    f[3] = axis + T(2) * g9 - (gu - T(4) * g4);
    f[2] = axis - g9 + g11 + (gv - T(4) * g6);
    f[4] = axis - g9 + g11 - (gv - T(4) * g6);
    f[9] = axis - g9 - g11 + (gw - T(4) * g8);
    f[14] = axis - g9 - g11 - (gw - T(4) * g8);
    const T dxy = diag + g9 + g11, dxz = diag + g9 - g11, dyz = diag - T(2) * g9;
    f[5] = dxy + g13 + (gu + gv + g4 + g6);
    f[7] = dxy + g13 - (gu + gv + g4 + g6);
    f[6] = dxy - g13 + (-gu + gv - g4 + g6);
    f[8] = dxy - g13 - (-gu + gv - g4 + g6);
    f[10] = dxz + g15 + (gu + gw + g4 + g8);
    f[17] = dxz + g15 - (gu + gw + g4 + g8);
    f[12] = dxz - g15 + (-gu + gw - g4 + g8);
    f[15] = dxz - g15 - (-gu + gw - g4 + g8);
    f[11] = dyz + g14 + (gv + gw + g6 + g8);
    f[18] = dyz + g14 - (gv + gw + g6 + g8);
    f[13] = dyz - g14 + (-gv + gw - g6 + g8);
    f[16] = dyz - g14 - (-gv + gw - g6 + g8);
}

/* Philox4x32-10 (Salmon et al., SC'11): counter (cell, step, 0, 0), key
 * (seed, 0); returns a uniform float in [0, 1) from the first output word.
 * Used for the seeded inlet noise, an extension the reference does not have. */
__host__ __device__ __forceinline__ float philox_uniform(uint32_t seed, uint32_t cell, uint32_t step) {
    uint32_t c0 = cell, c1 = step, c2 = 0u, c3 = 0u, k0 = seed, k1 = 0u;
#pragma unroll
    for (int r = 0; r < 10; ++r) {
        const uint64_t p0 = uint64_t(0xD2511F53u) * c0;
        const uint64_t p1 = uint64_t(0xCD9E8D57u) * c2;
        const uint32_t hi0 = uint32_t(p0 >> 32), lo0 = uint32_t(p0);
        const uint32_t hi1 = uint32_t(p1 >> 32), lo1 = uint32_t(p1);
        c0 = hi1 ^ c1 ^ k0;
        c1 = lo1;
        c2 = hi0 ^ c3 ^ k1;
        c3 = lo0;
        k0 += 0x9E3779B9u;
        k1 += 0xBB67AE85u;
    }
    return float(c0 >> 8) * (1.0f / 16777216.0f);
}

}  // namespace lbm
