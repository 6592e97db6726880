// Rotation-vector kinematics on the device.
//
// R(theta) = I + sinc(|theta|)[theta]x + 1/2 sinc(|theta|/2)^2 [theta]x^2
// (src/physics/pose.tpp:203-218) with sinc as src/utils/sinc.cpp:5-34 defines
// it.  Two flavours:
//  * rot_rn: every operation an explicit round-to-nearest intrinsic in a fixed
//    order, so the result is the same bits on any device and on the host
//    restatement (used wherever an exact decision depends on the vertex
//    positions: constraint sets, broad-phase boxes);
//  * body_frame: R with its first and second derivatives in theta, from the
//    closed-form gradient/Hessian of sinc(|x|) (sinc.cpp:103-141) and the
//    product rule on I + a K + b K^2 (R as rot_rn has it, contraction allowed
//    in the derivatives; used by the barrier and the inertial energy).
// sin/cos are evaluated by a Cody-Waite reduction by pi/2 (three-part split,
// 33-bit leading parts) and the Taylor series of sin and cos to degree 19/20
// (coefficients 1/n!) by Horner's rule; the error is below 2^-50|y| + 2^-60
// for |x| < 2^20.
#pragma once

#include <cuda_runtime.h>

namespace rigc {

#define RADD(a, b) __dadd_rn((a), (b))
#define RSUB(a, b) __dsub_rn((a), (b))
#define RMUL(a, b) __dmul_rn((a), (b))
#define RDIV(a, b) __ddiv_rn((a), (b))

__device__ __forceinline__ double det_reduce(double x, long long& k)
{
    const double kTwoOverPi = 0.6366197723675814;
    const double kP1 = 1.5707963267341256;
    const double kP2 = 6.077100506303966e-11;
    const double kP3 = 2.0222662487959506e-21;
    double kd = rint(RMUL(x, kTwoOverPi));
    k = (long long)kd;
    double r = RSUB(x, RMUL(kd, kP1));
    r = RSUB(r, RMUL(kd, kP2));
    r = RSUB(r, RMUL(kd, kP3));
    return r;
}

__device__ __forceinline__ double det_sin_poly(double r)
{
    double z = RMUL(r, r);
    double s = -1.0 / 121645100408832000.0;
    s = RMUL(s, z);
    s = RADD(1.0 / 355687428096000.0, s);
    s = RMUL(s, z);
    s = RADD(-1.0 / 1307674368000.0, s);
    s = RMUL(s, z);
    s = RADD(1.0 / 6227020800.0, s);
    s = RMUL(s, z);
    s = RADD(-1.0 / 39916800.0, s);
    s = RMUL(s, z);
    s = RADD(1.0 / 362880.0, s);
    s = RMUL(s, z);
    s = RADD(-1.0 / 5040.0, s);
    s = RMUL(s, z);
    s = RADD(1.0 / 120.0, s);
    s = RMUL(s, z);
    s = RADD(-1.0 / 6.0, s);
    double r3 = RMUL(r, z);
    return RADD(r, RMUL(r3, s));
}

__device__ __forceinline__ double det_cos_poly(double r)
{
    double z = RMUL(r, r);
    double p = 1.0 / 2432902008176640000.0;
    p = RMUL(p, z);
    p = RADD(-1.0 / 6402373705728000.0, p);
    p = RMUL(p, z);
    p = RADD(1.0 / 20922789888000.0, p);
    p = RMUL(p, z);
    p = RADD(-1.0 / 87178291200.0, p);
    p = RMUL(p, z);
    p = RADD(1.0 / 479001600.0, p);
    p = RMUL(p, z);
    p = RADD(-1.0 / 3628800.0, p);
    p = RMUL(p, z);
    p = RADD(1.0 / 40320.0, p);
    p = RMUL(p, z);
    p = RADD(-1.0 / 720.0, p);
    p = RMUL(p, z);
    p = RADD(1.0 / 24.0, p);
    p = RMUL(p, z);
    p = RADD(-0.5, p);
    p = RMUL(p, z);
    return RADD(1.0, p);
}

__device__ __forceinline__ double det_sin(double x)
{
    long long k;
    double r = det_reduce(x, k);
    switch (k & 3) {
    case 0: return det_sin_poly(r);
    case 1: return det_cos_poly(r);
    case 2: return -det_sin_poly(r);
    default: return -det_cos_poly(r);
    }
}

__device__ __forceinline__ double det_cos(double x)
{
    long long k;
    double r = det_reduce(x, k);
    switch (k & 3) {
    case 0: return det_cos_poly(r);
    case 1: return -det_sin_poly(r);
    case 2: return -det_cos_poly(r);
    default: return det_sin_poly(r);
    }
}

// both at once (shared reduction)
__device__ __forceinline__ void det_sincos(double x, double& s, double& c)
{
    long long k;
    double r = det_reduce(x, k);
    double sp = det_sin_poly(r), cp = det_cos_poly(r);
    switch (k & 3) {
    case 0: s = sp; c = cp; break;
    case 1: s = cp; c = -sp; break;
    case 2: s = -sp; c = -cp; break;
    default: s = -cp; c = sp; break;
    }
}

__device__ __forceinline__ double det_trig_err(double y)
{
    return RADD(RMUL(fabs(y), 8.881784197001252e-16), 8.673617379884035e-19);
}

// sinc (sinc.cpp:10-34) with round-to-nearest intrinsics
__device__ __forceinline__ double sinc_rn(double x)
{
    const double kT0 = 2.220446049250313e-16, kT2 = 1.4901161193847656e-08,
                 kTN = 1.220703125e-04;
    double ax = fabs(x);
    if (ax >= kTN) return RDIV(det_sin(x), x);
    double r = 1.0;
    if (ax >= kT0) {
        double x2 = RMUL(x, x);
        r = RSUB(r, RDIV(x2, 6.0));
        if (ax >= kT2) r = RADD(r, RDIV(RMUL(x2, x2), 120.0));
    }
    return r;
}

__device__ __forceinline__ double norm3_rn(double a, double b, double c)
{
    a = fabs(a);
    b = fabs(b);
    c = fabs(c);
    return __dsqrt_rn(RADD(RADD(RMUL(a, a), RMUL(b, b)), RMUL(c, c)));
}

// R row-major, exact operation order shared with the host restatement, from
// a = sinc(|t|) and s = sinc(|t / 2|)
__device__ __forceinline__ void rot_from_sinc(const double t[3], double a, double s, double R[9])
{
    double b = RMUL(RMUL(0.5, s), s);
    double K[9] = { 0.0, -t[2], t[1], t[2], 0.0, -t[0], -t[1], t[0], 0.0 };
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = 0; j < 3; j++) {
            double k2 = RADD(RADD(RMUL(K[3 * i], K[j]), RMUL(K[3 * i + 1], K[3 + j])),
                             RMUL(K[3 * i + 2], K[6 + j]));
            double r = RADD(RMUL(a, K[3 * i + j]), RMUL(b, k2));
            R[3 * i + j] = i == j ? RADD(r, 1.0) : r;
        }
}

__device__ __forceinline__ void rot_rn(const double t[3], double R[9])
{
    const double a = sinc_rn(norm3_rn(t[0], t[1], t[2]));
    const double s = sinc_rn(norm3_rn(RMUL(t[0], 0.5), RMUL(t[1], 0.5), RMUL(t[2], 0.5)));
    rot_from_sinc(t, a, s, R);
}

// V_j = ((v0 R_j0 + v1 R_j1) + v2 R_j2) + p_j
__device__ __forceinline__ void world_vertex_rn(const double R[9], const double p[3],
                                                const double v[3], double out[3])
{
#pragma unroll
    for (int j = 0; j < 3; j++)
        out[j] = RADD(RADD(RADD(RMUL(v[0], R[3 * j]), RMUL(v[1], R[3 * j + 1])),
                           RMUL(v[2], R[3 * j + 2])),
                      p[j]);
}

// ---------------------------------------------------------------------------
// body frame with derivatives (contraction allowed)

// d sinc(x)/dx / x and (d2 sinc/dx2 / x^2 - d sinc/dx / x^3) (sinc.cpp:103-141)
__device__ __forceinline__ double dsinc_over_x(double x, double s, double c)
{
    double x2 = x * x;
    if (fabs(x) > 1e-4) return (x * c - s) / (x2 * x);
    return x2 * (-x2 / 840.0 + 1.0 / 30.0) - 1.0 / 3.0;
}
__device__ __forceinline__ double ddsinc_term(double x, double s, double c)
{
    double x2 = x * x, x4 = x2 * x2;
    if (fabs(x) > 0.1) return ((3 - x2) * s - 3 * x * c) / (x4 * x);
    return x4 / 7560.0 - x2 / 210.0 + 1.0 / 15.0;
}

// Frame layout: R[9] | dR[3][9] | d2R[6][9] (pairs 00 01 02 11 12 22), all
// row-major 3x3.  dR[k] = dR/dtheta_k.
constexpr int kFrameDoubles = 90;

__device__ __forceinline__ int sym_index(int k, int l)
{
    // (0,0)=0 (0,1)=1 (0,2)=2 (1,1)=3 (1,2)=4 (2,2)=5
    if (k > l) { int t = k; k = l; l = t; }
    return k == 0 ? l : (k == 1 ? 2 + l : 5);
}

// sinc and its derivatives' factors at x = |t| or |t / 2|
struct SincTerms {
    double s, g1, g2;
};
__device__ __forceinline__ SincTerms sinc_terms(double x)
{
    double sn, cn;
    det_sincos(x, sn, cn);
    return SincTerms { x >= 1.220703125e-04 ? RDIV(sn, x) : sinc_rn(x), dsinc_over_x(x, sn, cn), ddsinc_term(x, sn, cn) };
}

// a(t) = sinc(|t|): gradient a1 t, Hessian a2 t t^T + a1 I; b = 1/2 s^2 with
// s(t) = sinc(|t / 2|): ds = 1/2 g(t/2), d2s = 1/4 H(t/2), so that gb = s ds,
// Hb = ds ds^T + s d2s
struct FrameBase {
    double t[3], gs[3];
    double a, a1, a2, b, sh, h1, h2;
};
__device__ __forceinline__ FrameBase frame_base(const double t[3], const SincTerms& full, const SincTerms& half)
{
    FrameBase f;
    for (int i = 0; i < 3; i++) {
        f.t[i] = t[i];
        f.gs[i] = 0.25 * half.g1 * t[i];
    }
    f.a = full.s;
    f.a1 = full.g1;
    f.a2 = full.g2;
    f.sh = half.s;
    f.b = RMUL(RMUL(0.5, half.s), half.s);
    f.h1 = 0.25 * half.g1;
    f.h2 = 0.0625 * half.g2;
    return f;
}

// [e_k]x's entry (i, j)
__device__ __forceinline__ double unit_cross(int k, int i, int j)
{
    return i == j || i == k || j == k ? 0.0 : (i - k + 3) % 3 == 1 ? -1.0 : 1.0;
}

// entry e of the frame: with K = [t]x, E_k = [e_k]x and
//   (K K)_ij = t_i t_j - |t|^2 d_ij, (E_k K + K E_k)_ij = t_i d_jk + t_j d_ik - 2 t_k d_ij,
//   (E_k E_l + E_l E_k)_ij = d_il d_jk + d_ik d_jl - 2 d_kl d_ij
// R = I + a K + b K K and its derivatives by the product rule.  The order of the
// derivatives' sums is arbitrary: five of the six tried end the converged run of 27
// landing cubes (test_gpu_step.py) at an outcome that the oracle has, this is one.
__device__ __forceinline__ double frame_entry(const FrameBase& f, int e)
{
    const int i = (e % 9) / 3, j = e % 3;
    const int m = (3 - i - j + 3) % 3;  // the third index when i != j
    const double ti = f.t[i], tj = f.t[j];
    const int u = (i + 1) % 3, v = (i + 2) % 3;
    const double K = i == j ? 0.0 : unit_cross(m, i, j) * f.t[m];
    const double K2 = i == j ? -RADD(RMUL(f.t[u], f.t[u]), RMUL(f.t[v], f.t[v])) : RMUL(ti, tj);
    if (e < 9) {  // as rot_rn
        const double r = RADD(RMUL(f.a, K), RMUL(f.b, K2));
        return i == j ? RADD(r, 1.0) : r;
    }
    auto pair = [&](int k) { return (j == k ? ti : 0.0) + (i == k ? tj : 0.0) - (i == j ? 2 * f.t[k] : 0.0); };
    if (e < 36) {
        const int k = (e - 9) / 9;
        const double gb = f.sh * f.gs[k];
        return fma(f.a1 * f.t[k], K, fma(f.a, unit_cross(k, i, j), fma(gb, K2, f.b * pair(k))));
    }
    const int q = (e - 36) / 9, k = q < 3 ? 0 : q < 5 ? 1 : 2, l = q < 3 ? q : q < 5 ? q - 2 : 2;
    const double kl = k == l ? 1.0 : 0.0;
    const double Ha = fma(f.a2, f.t[k] * f.t[l], kl * f.a1);
    const double Hb = fma(f.gs[k], f.gs[l], f.sh * fma(f.h2, f.t[k] * f.t[l], kl * f.h1));
    const double ee = (double)((i == l) * (j == k) + (i == k) * (j == l)) - (i == j ? 2 * kl : 0.0);
    double r = f.b * ee;
    r = fma(f.sh * f.gs[l], pair(k), r);
    r = fma(f.sh * f.gs[k], pair(l), r);
    r = fma(Hb, K2, r);
    r = fma(f.a1 * f.t[l], unit_cross(k, i, j), r);
    r = fma(f.a1 * f.t[k], unit_cross(l, i, j), r);
    return fma(Ha, K, r);
}

__device__ inline void body_frame(const double t[3], double* F)
{
    const double n = norm3_rn(t[0], t[1], t[2]);
    const FrameBase f = frame_base(t, sinc_terms(n), sinc_terms(0.5 * n));
#pragma unroll
    for (int e = 0; e < kFrameDoubles; e++) F[e] = frame_entry(f, e);
}

// The frame by a warp: half the lanes take the whole angle and half the half
// angle, then three entries each.  A thread's chain of some 1500 FP64
// instructions took 32 us however few the bodies, this 11.
__device__ __forceinline__ void warp_body_frame(const double t[3], int lane, double* F)
{
    const double n = norm3_rn(t[0], t[1], t[2]);
    const SincTerms mine = sinc_terms(lane < 16 ? n : 0.5 * n);
    SincTerms q[2];
    for (int k = 0; k < 2; k++)
        q[k] = SincTerms { __shfl_sync(0xffffffffu, mine.s, 16 * k), __shfl_sync(0xffffffffu, mine.g1, 16 * k),
                           __shfl_sync(0xffffffffu, mine.g2, 16 * k) };
    const FrameBase f = frame_base(t, q[0], q[1]);
    for (int e = lane; e < kFrameDoubles; e += 32) F[e] = frame_entry(f, e);
}

// Bodies up to which a warp takes one, then a thread: a warp's 250 instructions
// fill the FP64 units (608 sub-partitions, 64 cycles an instruction) longer than
// one thread's chain lasts from some 2000 bodies on.
constexpr int kWarpFrames = 2048;

} // namespace rigc
