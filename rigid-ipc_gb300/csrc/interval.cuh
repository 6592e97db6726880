// Interval arithmetic on the device for the rigid CCD.
//
// Semantics of the reference's Interval (src/interval/interval.hpp:25-30):
// Boost.Interval operations over the FILibRounding policy
// (src/interval/filib_rounding.cpp:12-60), i.e. each bound is the
// round-to-nearest result stepped one ulp outward, with exact-zero results
// kept exact (x == -y for sums, x == y for differences, a zero factor for
// products, a zero dividend for quotients).  Products and quotients use the
// sign-case tables; widths round up; cos/sin reduce by an enclosure of 2*pi and
// evaluate the monotone pieces with the deterministic cosine of rotation.cuh
// widened by its error bound.  The ulp steps are integer operations on the
// bit pattern.
#pragma once

#include "rotation.cuh"

namespace rigc {

struct Itv {
    double lo, hi;
};

__device__ __forceinline__ Itv mk(double l, double h) { return Itv { l, h }; }
__device__ __forceinline__ Itv pt(double x) { return Itv { x, x }; }
__device__ __forceinline__ Itv iempty()
{
    return Itv { __longlong_as_double(0x7ff8000000000000ll), __longlong_as_double(0x7ff8000000000000ll) };
}
__device__ __forceinline__ bool is_empty(const Itv& x) { return !(x.lo <= x.hi); }

// Bit pattern of a double through an opaque move: the optimizer cannot turn
// the integer tests below back into double-precision compares.
__device__ __forceinline__ long long dbits(double x)
{
    long long r;
    asm("mov.b64 %0, %1;" : "=l"(r) : "d"(x));
    return r;
}

// next double towards -inf / +inf (nextafter semantics, finite and zero inputs)
__device__ __forceinline__ double dpred(double x)
{
    long long b = dbits(x);
    if ((b & 0x7fffffffffffffffll) == 0) return __longlong_as_double(0x8000000000000001ll);
    if (b == (long long)0xfff0000000000000ull) return x;
    return __longlong_as_double(b > 0 ? b - 1 : b + 1);
}
__device__ __forceinline__ double dsucc(double x)
{
    long long b = dbits(x);
    if ((b & 0x7fffffffffffffffll) == 0) return __longlong_as_double(1ll);
    if (b == 0x7ff0000000000000ll) return x;
    return __longlong_as_double(b > 0 ? b + 1 : b - 1);
}

// Sign and order tests on the bit pattern (integer instructions; the
// double-precision pipe is the scarce one on this GPU).  Exact for every
// non-NaN double, +-0 and +-inf included; no NaN reaches them.
__device__ __forceinline__ bool is_zero(double x) { return (dbits(x) << 1) == 0; }
// x < 0: sign bit set and not -0
__device__ __forceinline__ bool is_neg(double x)
{
    return (unsigned long long)dbits(x) > 0x8000000000000000ull;
}
// x > 0
__device__ __forceinline__ bool is_pos(double x) { return dbits(x) > 0; }
// monotone integer key: key(x) < key(y) iff x < y, except -0 < +0
__device__ __forceinline__ long long order_key(double x)
{
    long long b = dbits(x);
    return b ^ ((b >> 63) & 0x7fffffffffffffffll);
}
// x < y
__device__ __forceinline__ bool lt(double x, double y)
{
    return order_key(x) < order_key(y) && !(is_zero(x) && is_zero(y));
}

// A sum or difference of finite doubles is zero only when exact (no
// underflow to zero), so the exact-zero rule tests the rounded result.
__device__ __forceinline__ double add_dn(double x, double y)
{
    double r = RADD(x, y);
    return is_zero(r) ? 0.0 : dpred(r);
}
__device__ __forceinline__ double add_up(double x, double y)
{
    double r = RADD(x, y);
    return is_zero(r) ? 0.0 : dsucc(r);
}
__device__ __forceinline__ double sub_dn(double x, double y)
{
    double r = RSUB(x, y);
    return is_zero(r) ? 0.0 : dpred(r);
}
__device__ __forceinline__ double sub_up(double x, double y)
{
    double r = RSUB(x, y);
    return is_zero(r) ? 0.0 : dsucc(r);
}
__device__ __forceinline__ double mul_dn(double x, double y)
{
    return (is_zero(x) || is_zero(y)) ? 0.0 : dpred(RMUL(x, y));
}
__device__ __forceinline__ double mul_up(double x, double y)
{
    return (is_zero(x) || is_zero(y)) ? 0.0 : dsucc(RMUL(x, y));
}
__device__ __forceinline__ double div_dn(double x, double y) { return is_zero(x) ? 0.0 : dpred(RDIV(x, y)); }
__device__ __forceinline__ double div_up(double x, double y) { return is_zero(x) ? 0.0 : dsucc(RDIV(x, y)); }

__device__ __forceinline__ double smin(double a, double b) { return lt(b, a) ? b : a; }
__device__ __forceinline__ double smax(double a, double b) { return lt(a, b) ? b : a; }

__device__ __forceinline__ Itv ineg(const Itv& x) { return Itv { -x.hi, -x.lo }; }
__device__ __forceinline__ Itv iadd(const Itv& x, const Itv& y)
{
    return Itv { add_dn(x.lo, y.lo), add_up(x.hi, y.hi) };
}
__device__ __forceinline__ Itv iadd(double x, const Itv& y) { return Itv { add_dn(x, y.lo), add_up(x, y.hi) }; }
__device__ __forceinline__ Itv isub(const Itv& x, const Itv& y)
{
    return Itv { sub_dn(x.lo, y.hi), sub_up(x.hi, y.lo) };
}
__device__ __forceinline__ Itv isub(const Itv& x, double y) { return Itv { sub_dn(x.lo, y), sub_up(x.hi, y) }; }

__device__ __forceinline__ Itv imul(const Itv& x, const Itv& y)
{
    const double xl = x.lo, xu = x.hi, yl = y.lo, yu = y.hi;
    if (is_neg(xl)) {
        if (is_pos(xu)) {
            if (is_neg(yl)) {
                if (is_pos(yu))
                    return Itv { smin(mul_dn(xl, yu), mul_dn(xu, yl)), smax(mul_up(xl, yl), mul_up(xu, yu)) };
                return Itv { mul_dn(xu, yl), mul_up(xl, yl) };
            }
            if (is_pos(yu)) return Itv { mul_dn(xl, yu), mul_up(xu, yu) };
            return Itv { 0.0, 0.0 };
        }
        if (is_neg(yl)) {
            if (is_pos(yu)) return Itv { mul_dn(xl, yu), mul_up(xl, yl) };
            return Itv { mul_dn(xu, yu), mul_up(xl, yl) };
        }
        if (is_pos(yu)) return Itv { mul_dn(xl, yu), mul_up(xu, yl) };
        return Itv { 0.0, 0.0 };
    }
    if (is_pos(xu)) {
        if (is_neg(yl)) {
            if (is_pos(yu)) return Itv { mul_dn(xu, yl), mul_up(xu, yu) };
            return Itv { mul_dn(xu, yl), mul_up(xl, yu) };
        }
        if (is_pos(yu)) return Itv { mul_dn(xl, yl), mul_up(xu, yu) };
        return Itv { 0.0, 0.0 };
    }
    return Itv { 0.0, 0.0 };
}

// Product with an interval y whose lower bound is not negative (time and
// barycentric intervals): the sign-case table reduces to one choice of
// factor per bound, made without branches.
__device__ __forceinline__ Itv imul_nonneg(const Itv& x, const Itv& y)
{
    const double yl = is_neg(x.lo) ? y.hi : y.lo;
    const double yu = is_neg(x.hi) ? y.lo : y.hi;
    return Itv { mul_dn(x.lo, yl), mul_up(x.hi, yu) };
}

// scalar times interval (a zero scalar gives [0, 0] through the zero rule)
__device__ __forceinline__ Itv imul(double x, const Itv& y)
{
    const bool neg = is_neg(x);
    return Itv { mul_dn(x, neg ? y.hi : y.lo), mul_up(x, neg ? y.lo : y.hi) };
}

// quotient by an interval that excludes zero (the only case on this path)
__device__ __forceinline__ Itv idiv(const Itv& x, const Itv& y)
{
    const double xl = x.lo, xu = x.hi, yl = y.lo, yu = y.hi;
    if (yl <= 0 && yu >= 0) {
        if (xl == 0 && xu == 0) return Itv { 0.0, 0.0 };
        return Itv { -INFINITY, INFINITY };
    }
    if (is_neg(xu)) {
        if (is_neg(yu)) return Itv { div_dn(xu, yl), div_up(xl, yu) };
        return Itv { div_dn(xl, yl), div_up(xu, yu) };
    }
    if (is_neg(xl)) {
        if (is_neg(yu)) return Itv { div_dn(xu, yu), div_up(xl, yu) };
        return Itv { div_dn(xl, yl), div_up(xu, yl) };
    }
    if (is_neg(yu)) return Itv { div_dn(xu, yu), div_up(xl, yl) };
    return Itv { div_dn(xl, yu), div_up(xu, yl) };
}
__device__ __forceinline__ Itv idiv(const Itv& x, double y)
{
    if (is_neg(y)) return Itv { div_dn(x.hi, y), div_up(x.lo, y) };
    return Itv { div_dn(x.lo, y), div_up(x.hi, y) };
}

__device__ __forceinline__ Itv isqrt(const Itv& x)
{
    if (is_empty(x) || is_neg(x.hi)) return iempty();
    double l = !is_pos(x.lo) ? 0.0 : (x.lo == 0 ? 0.0 : dpred(__dsqrt_rn(x.lo)));
    double h = x.hi == 0 ? 0.0 : dsucc(__dsqrt_rn(x.hi));
    return Itv { l, h };
}

__device__ __forceinline__ Itv iabs(const Itv& x)
{
    if (!is_neg(x.lo)) return x;
    if (!is_pos(x.hi)) return ineg(x);
    return Itv { 0.0, smax(-x.lo, x.hi) };
}

__device__ __forceinline__ Itv ihull(const Itv& x, const Itv& y)
{
    if (is_empty(x)) return y;
    if (is_empty(y)) return x;
    return Itv { smin(x.lo, y.lo), smax(x.hi, y.hi) };
}

__device__ __forceinline__ bool zero_in(const Itv& x) { return !is_pos(x.lo) && !is_neg(x.hi); }
__device__ __forceinline__ double iwidth(const Itv& x) { return sub_up(x.hi, x.lo); }

// ---------------------------------------------------------------------------
// cos / sin

constexpr double kPiLo = 3.141592653589793116;
constexpr double kPiHi = 3.141592653589793560;

__device__ __forceinline__ double clamp_pm1(double r) { return r < -1.0 ? -1.0 : (r > 1.0 ? 1.0 : r); }

__device__ __forceinline__ double cos_dn(double x)
{
    if (fabs(x) > 1048576.0) return -1.0;
    double c = det_cos(x);
    return clamp_pm1(dpred(RSUB(c, det_trig_err(c))));
}
__device__ __forceinline__ double cos_up(double x)
{
    if (fabs(x) > 1048576.0) return 1.0;
    double c = det_cos(x);
    return clamp_pm1(dsucc(RADD(c, det_trig_err(c))));
}

// x - n [lo, hi](2 pi) with n = floor(div_dn(x.lo, 2 pi)).  A product with the
// reciprocal gives the same n wherever it is further from an integer than its
// error (the quotient takes some 12 double-precision instructions).
__device__ __forceinline__ Itv ifmod(const Itv& x, const Itv& y)
{
    const double q = RMUL(x.lo, 0.15915494309189535);
    double n = floor(q);
    const double f = RSUB(q, n);
    if (!(fabs(q) < 1024.0 && f > 1e-9 && f < 1.0 - 1e-9)) n = floor(div_dn(x.lo, is_neg(x.lo) ? y.lo : y.hi));
    return isub(x, imul(n, y));
}

// one bound of the cosine over x
static __device__ __noinline__ double icos_bound(Itv x, bool upper)
{
    const Itv pi2 { kPiLo * 2, kPiHi * 2 };
    bool negate = false, none = false;
    Itv tmp;
    for (int pass = 0; pass < 2; pass++) {
        tmp = ifmod(x, pi2);
        none = iwidth(tmp) >= pi2.lo;
        if (none || negate || !(tmp.lo >= kPiHi)) break;
        x = isub(tmp, Itv { kPiLo, kPiHi });
        negate = true;
    }
    const bool up = upper != negate;
    double r = up ? 1.0 : -1.0;
    if (!none && (up ? tmp.hi <= pi2.lo : tmp.hi <= kPiLo)) {
        const double at = !up ? tmp.hi : tmp.hi <= kPiLo ? tmp.lo : smin(sub_dn(pi2.lo, tmp.hi), tmp.lo);
        r = up ? cos_up(at) : cos_dn(at);
    }
    return negate ? -r : r;
}

__device__ __forceinline__ double isin_bound(const Itv& x, bool upper)
{
    return icos_bound(isub(x, Itv { kPiLo / 2, kPiHi / 2 }), upper);
}

// one bound of sinc at a point >= 0 (sinc.cpp:36-47)
static __device__ __noinline__ double sinc_bound(double xd, bool upper)
{
    const Itv x = pt(xd);
    if (xd >= 1.220703125e-04) {
        const double s = isin_bound(x, upper);
        return upper ? div_up(s, xd) : div_dn(s, xd);
    }
    const Itv x2 = imul(x, x);
    const Itv t = iadd(1.0, imul(idiv(x2, 6.0), isub(idiv(x2, 20.0), 1.0)));
    return upper ? t.hi : t.lo;
}

constexpr double kSincMono = 4.4934094579;  // sinc decreases up to here

// sinc over a non-negative interval (sinc.cpp:49-101; the input is a norm)
static __device__ __noinline__ Itv isinc_nonneg(const Itv& x)
{
    Itv y = iempty();
    Itv x_gt = x;
    if (x.lo <= kSincMono) {
        Itv x_mono = x;
        if (x_mono.hi > kSincMono) {
            x_mono = Itv { x_mono.lo, kSincMono };
            x_gt = Itv { kSincMono, x.hi };
        } else {
            x_gt = iempty();
        }
        y = Itv { smax(sinc_bound(x_mono.hi, false), -0.271724), smin(sinc_bound(x_mono.lo, true), 1.0) };
    }
    if (!is_empty(x_gt)) y = ihull(y, idiv(Itv { isin_bound(x_gt, false), isin_bound(x_gt, true) }, x_gt));
    return y;
}

// one bound of it
__device__ __forceinline__ double isinc_nonneg_bound(const Itv& x, bool upper)
{
    if (x.lo <= kSincMono && x.hi <= kSincMono) {
        const double b = sinc_bound(upper ? x.lo : x.hi, upper);
        return upper ? smin(b, 1.0) : smax(b, -0.271724);
    }
    const Itv y = isinc_nonneg(x);
    return upper ? y.hi : y.lo;
}

__device__ __forceinline__ Itv inorm(const Itv r[3])
{
    Itv a0 = iabs(r[0]), a1 = iabs(r[1]), a2 = iabs(r[2]);
    return isqrt(iadd(iadd(imul(a0, a0), imul(a1, a1)), imul(a2, a2)));
}

__device__ __forceinline__ Itv isinc_norm(const Itv r[3]) { return isinc_nonneg(inorm(r)); }

// 0 + x: the bounds one step outward
__device__ __forceinline__ Itv istep(const Itv& x)
{
    return Itv { is_zero(x.lo) ? 0.0 : dpred(x.lo), is_zero(x.hi) ? 0.0 : dsucc(x.hi) };
}

// Interval rotation matrix (pose.tpp:203-218), row-major: sa K + c K K + I,
// each sum (K K)_ij = K_i0 K_0j + (K_i1 K_1j + K_i2 K_2j).  Bound by FP64 issue
// (an interval frame was some 820 double-precision instructions): the bounds of
// the two sinc are evaluated one by one, as only one of each end's is used (8
// -> 4 cosines and divisions); K's zeros leave only the outward step of a sum;
// the products that K's antisymmetry makes equal (each bound is the same
// rounded product) are taken once; halves are products.  Same bits.  Frames of
// 1000 bodies over 128 time nodes each: 411 -> 201 us.
static __device__ __noinline__ void irotation(const Itv r[3], Itv R[9])
{
    const Itv sa = isinc_norm(r);
    Itv rh[3];
#pragma unroll
    for (int k = 0; k < 3; k++) rh[k] = Itv { mul_dn(r[k].lo, 0.5), mul_up(r[k].hi, 0.5) };
    const Itv sh = isinc_norm(rh);
    const Itv c = imul(imul(0.5, sh), sh);
    Itv n[3], s[3];  // -r_k r_k (as independent factors), sa r_k
#pragma unroll
    for (int k = 0; k < 3; k++) {
        n[k] = imul(ineg(r[k]), r[k]);
        s[k] = imul(sa, r[k]);
    }
    const Itv d[3] = { istep(iadd(n[2], n[1])), iadd(n[2], istep(n[0])), iadd(n[1], istep(n[0])) };
#pragma unroll
    for (int k = 0; k < 3; k++) R[4 * k] = iadd(istep(imul(c, d[k])), pt(1.0));
    const Itv m01 = imul(c, istep(istep(imul(r[1], r[0])))), m02 = imul(c, istep(istep(imul(r[2], r[0])))),
              m12 = imul(c, istep(imul(r[2], r[1])));
    R[1] = iadd(ineg(s[2]), m01);
    R[3] = iadd(s[2], m01);
    R[2] = iadd(s[1], m02);
    R[6] = iadd(ineg(s[1]), m02);
    R[5] = iadd(ineg(s[0]), m12);
    R[7] = iadd(s[0], m12);
}

// The same by four lanes (q = 0 .. 3): a bound of the two sinc each, then lane k
// < 3 the entries of R's diagonal and of K at index k
__device__ __forceinline__ void irotation_quad(const Itv r[3], int q, Itv* diag, Itv* neg, Itv* pos)
{
    Itv x[3];
#pragma unroll
    for (int k = 0; k < 3; k++) x[k] = q < 2 ? r[k] : Itv { mul_dn(r[k].lo, 0.5), mul_up(r[k].hi, 0.5) };
    const double b = isinc_nonneg_bound(inorm(x), q & 1);
    const Itv sa { __shfl_sync(0xffffffffu, b, 0, 4), __shfl_sync(0xffffffffu, b, 1, 4) };
    const Itv sh { __shfl_sync(0xffffffffu, b, 2, 4), __shfl_sync(0xffffffffu, b, 3, 4) };
    const Itv c = imul(imul(0.5, sh), sh);
    const Itv ru = q == 2 ? r[1] : r[2], rv = q == 0 ? r[1] : r[0], rk = q == 0 ? r[0] : q == 1 ? r[1] : r[2];
    const Itv nu = imul(ineg(ru), ru), nv = imul(ineg(rv), rv);
    const Itv d = q == 0 ? istep(iadd(nu, nv)) : iadd(nu, istep(nv));
    *diag = iadd(istep(imul(c, d)), pt(1.0));
    Itv t = istep(imul(ru, rv));
    if (q > 0) t = istep(t);
    const Itv m = imul(c, t), s = imul(sa, rk);
    *neg = iadd(ineg(s), m);
    *pos = iadd(s, m);
}

// world vertex over intervals: ((v0 R_j0 + v1 R_j1) + v2 R_j2) + p_j
__device__ __forceinline__ void iworld_vertex(const Itv R[9], const Itv p[3], const double v[3],
                                              Itv out[3])
{
#pragma unroll
    for (int j = 0; j < 3; j++)
        out[j] = iadd(iadd(iadd(imul(v[0], R[3 * j]), imul(v[1], R[3 * j + 1])),
                           imul(v[2], R[3 * j + 2])),
                      p[j]);
}

} // namespace rigc
