// The two-degree Legendre recurrence of the grid transforms (K. Ishioka,
// J. Meteorol. Soc. Japan 96, 2018): with n = m + 2 l + 1 and
// eps_n = sqrt((n^2 - m^2) / (4 n^2 - 1)) the functions
//     q_l = P_n,m / sin(lat)
// are polynomials in x2 = sin^2(lat) (times cos^m) with
//     q_l+1 eps_n+1 eps_n+2 = (x2 - eps_n+1^2 - eps_n^2) q_l
//                             - eps_n eps_n-1 q_l-1,
// and q_l = k_l s_l with k_l+1 / k_l-1 = eps_n eps_n-1 / (eps_n+1 eps_n+2)
// turns that into
//     s_l+1 = (alpha_l x2 + beta_l) s_l - s_l-1,                        (1)
// two fused operations for two degrees.  Both parities follow from q:
//     P_m+2l+1 = x q_l,   P_m+2l = eps_m+2l+1 q_l + eps_m+2l q_l-1,
// so the sums over even degrees are sums over q with the coefficients
// combined in pairs (two_tables.cu), and the odd ones take one product by
// sin(lat) at the end.  Per (degree, order, latitude pair) three FP64
// instructions instead of the four of leg.cuh's one-degree recurrence, and
// only one of the six per two degrees reads three registers that no
// neighbouring instruction reads (such a DFMA runs at 12.3 T lanes/s on
// B200, one that shares an operand with its neighbours at up to 18.3).
//
// Rounding.  x2 must be exact to half an ulp of its own size, not the square
// of a rounded sine: its error acts as a constant shift of the latitude.
// (1) takes it as x2 near the equator and as gamma_l - alpha_l u2 (gamma =
// alpha + beta, u2 = cos^2) towards the poles, each from double-double
// (k_geometry).  Against 80-bit functions of the true latitude, relative RMS
// over the latitudes of the nmax 2190 grid: 2.1e-14 (m = 0), 1.6e-14 (500),
// 1.2e-14 (1500), where leg.cuh's recurrence gives 8.0e-14, 4.9e-14,
// 2.3e-14.  Within |sin(lat)| < TWO_NEAR the even functions are small
// differences of the q's; those latitudes stay with the one-degree
// recurrence (without them here: 5.0e-14, 3.0e-14, 1.6e-14).
//
// s_l and k_l vary slowly, so no multipliers at chunk boundaries; values far
// below the double range carry a binary exponent as in leg.cuh.
#pragma once

#include "common.cuh"
#include "kernels.h"
#include "leg.cuh"

namespace cb
{

constexpr int TWO_CHUNK = 32;   // steps (of two degrees) per staged chunk

// number of steps of order m up to degree nmax
__host__ __device__ __forceinline__ long long two_len(long long nmax,
                                                      long long m)
{
    return (nmax - m) / 2 + 1;
}

// first step of order m in order-major arrays of degree nmax
__host__ __device__ __forceinline__ long long two_col0(long long nmax,
                                                       long long m)
{
    return two_sum(nmax) - two_sum(nmax - m);
}

// ---------------------------------------------------------------------------
// Sectorial seeds and scaled latitudes.  u^m of every pair is the product of
// two entries of a table that k_geometry fills per call (u^r, r < 64, and
// u^(64 j), each (mantissa, binary exponent) from the double-double cosine):
// one product instead of the 2 log2(m) dependent ones of pow_me, which were
// a third of the kernel's instructions at nmax 2190.
// ---------------------------------------------------------------------------
// 2^e for -1022 <= e <= 1023
__device__ __forceinline__ double pow2i(int e)
{
    return __hiloint2double((e + 1023) << 20, 0);
}

// Normalises a scaled state as leg_fixup does (true when the latitude turned
// unscaled), with products by powers of two in place of scalbn.  A chunk of
// TWO_CHUNK steps multiplies the state by at most the 64 first factors
// 1 / eps_m+i of its order, about ((2 m)^64 / 64!)^(1/2): 2^313 at m = 10800,
// 2^402 at the largest order that the row transforms serve.  So a latitude
// turns with E above -1000 up to m = 10800; beyond, where E is no exponent of
// a double yet, it turns one chunk later (what it then leaves out is below
// 2^-198).
__device__ __forceinline__ bool two_fixup(double &x, double &y, int &E)
{
    if (E == 0)
        return false;
    const int ex = (__double2hiint(x) >> 20) & 0x7ff;
    const int ey = (__double2hiint(y) >> 20) & 0x7ff;
    const int e = max(ex, ey) - 1023;
    if (e == -1023 || e == 1024)
        return false;
    const int tot = E + e;
    const bool back = tot >= LEG_SWITCH_EXP && E > -1000;
    const double f = pow2i(back ? E : -e);
    x *= f;
    y *= f;
    E = back ? 0 : tot;
    return back;
}

// Seed sigma u^m of pair p, normalised.
__device__ __forceinline__ void two_seed(const double2 *pw, long long np,
                                         long long p, long long m,
                                         double sigma, double &x, int &E)
{
    const double2 a = pw[(m & (POW_LOW - 1)) * np + p];
    const double2 b = pw[(POW_LOW + m / POW_LOW) * np + p];
    x = sigma * (a.x * b.x);
    E = (int)(a.y + b.y);
    const int e = ((__double2hiint(x) >> 20) & 0x7ff) - 1023;
    if (e == -1023)
        E = 0;
    else if (E + e >= LEG_SWITCH_EXP)
    {
        x *= pow2i(E);
        E = 0;
    }
    else
    {
        x *= pow2i(-e);
        E += e;
    }
}

// double-double arithmetic (Dekker / Knuth with fused products)
struct dd
{
    double hi, lo;
};

__device__ __forceinline__ dd dd_fast(double a, double b)
{
    const double s = a + b;
    return {s, b - (s - a)};
}

__device__ __forceinline__ dd dd_add(dd a, dd b)
{
    const double s = a.hi + b.hi;
    const double v = s - a.hi;
    const double e = (a.hi - (s - v)) + (b.hi - v);
    return dd_fast(s, e + (a.lo + b.lo));
}

__device__ __forceinline__ dd dd_mul(dd a, dd b)
{
    const double p = a.hi * b.hi;
    const double e = fma(a.hi, b.hi, -p);
    return dd_fast(p, fma(a.hi, b.lo, fma(a.lo, b.hi, e)));
}

__device__ __forceinline__ dd dd_neg(dd a) { return {-a.hi, -a.lo}; }

__device__ __forceinline__ dd dd_div(dd a, dd b)
{
    const double q = a.hi / b.hi;
    const dd r = dd_add(a, dd_neg(dd_mul(b, dd{q, 0.0})));
    return dd_fast(q, r.hi / b.hi);
}

__device__ __forceinline__ dd dd_sqrt(dd a)
{
    const double q = sqrt(a.hi);
    const dd r = dd_add(a, dd_neg(dd_mul(dd{q, 0.0}, dd{q, 0.0})));
    return dd_fast(q, r.hi / (2.0 * q));
}

} // namespace cb
