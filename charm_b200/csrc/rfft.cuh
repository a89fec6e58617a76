// Device code of the row transforms (rfft.cu describes them), shared by
// rfft.cu and the files that compile the one-CTA kernels of some plans each
// (rfft_ct*.cu).
#pragma once

#include <cstdint>
#include <type_traits>

#include <cooperative_groups.h>

#include "common.cuh"
#include "kernels.h"

namespace cb
{

namespace
{

__device__ __forceinline__ double2 cmul(double2 a, double2 b)
{
    return make_double2(fma(a.x, b.x, -a.y * b.y), fma(a.x, b.y, a.y * b.x));
}

__device__ __forceinline__ double2 conj2(double2 a)
{
    return make_double2(a.x, -a.y);
}

__device__ __forceinline__ double2 add2(double2 a, double2 b)
{
    return make_double2(a.x + b.x, a.y + b.y);
}

__device__ __forceinline__ double2 sub2(double2 a, double2 b)
{
    return make_double2(a.x - b.x, a.y - b.y);
}

// -i a
__device__ __forceinline__ double2 mul_mi(double2 a)
{
    return make_double2(a.y, -a.x);
}

// shared-memory position of element i
__device__ __forceinline__ int pidx(int i)
{
    return i + (i >> 3);
}

constexpr double RSQRT2 = 0.70710678118654752440;
constexpr double SQRT3_2 = 0.86602540378443864676;

// In-register forward DFTs, X_k = sum_r v_r exp(-2 pi i r k / R).
__device__ __forceinline__ void dft2(double2 *v)
{
    double2 a = v[0], b = v[1];
    v[0] = add2(a, b);
    v[1] = sub2(a, b);
}

__device__ __forceinline__ void dft4(double2 &a0, double2 &a1, double2 &a2,
                                     double2 &a3)
{
    double2 t0 = add2(a0, a2), t1 = sub2(a0, a2);
    double2 t2 = add2(a1, a3), t3 = mul_mi(sub2(a1, a3));
    a0 = add2(t0, t2);
    a2 = sub2(t0, t2);
    a1 = add2(t1, t3);
    a3 = sub2(t1, t3);
}

__device__ __forceinline__ void dft8(double2 *v)
{
    // even / odd halves, then one radix-2 step with W8^k
    double2 e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6];
    double2 o0 = v[1], o1 = v[3], o2 = v[5], o3 = v[7];
    dft4(e0, e1, e2, e3);
    dft4(o0, o1, o2, o3);
    double2 w1 = make_double2((o1.x + o1.y) * RSQRT2, (o1.y - o1.x) * RSQRT2);
    double2 w2 = mul_mi(o2);
    double2 w3 = make_double2((o3.y - o3.x) * RSQRT2, -(o3.x + o3.y) * RSQRT2);
    v[0] = add2(e0, o0);
    v[4] = sub2(e0, o0);
    v[1] = add2(e1, w1);
    v[5] = sub2(e1, w1);
    v[2] = add2(e2, w2);
    v[6] = sub2(e2, w2);
    v[3] = add2(e3, w3);
    v[7] = sub2(e3, w3);
}

__device__ __forceinline__ void dft3(double2 *v)
{
    double2 t = add2(v[1], v[2]);
    double2 d = sub2(v[1], v[2]);
    double2 h = make_double2(fma(-0.5, t.x, v[0].x), fma(-0.5, t.y, v[0].y));
    double2 q = mul_mi(make_double2(SQRT3_2 * d.x, SQRT3_2 * d.y));
    v[0] = add2(v[0], t);
    v[1] = add2(h, q);
    v[2] = sub2(h, q);
}

// cos and sin of pi/8, 2 pi/9, 4 pi/9, 8 pi/9
constexpr double C16 = 0.92387953251128675613;
constexpr double S16 = 0.38268343236508977173;
constexpr double C9A = 0.76604444311897803520;
constexpr double S9A = 0.64278760968653932632;
constexpr double C9B = 0.17364817766693034885;
constexpr double S9B = 0.98480775301220805936;
constexpr double C9D = -0.93969262078590838405;
constexpr double S9D = 0.34202014332566873304;

// 16 = 4 x 4 (n = 4 n1 + n2, k = k1 + 4 k2): DFTs of length 4 over n1,
// twiddles exp(-2 pi i n2 k1 / 16), DFTs of length 4 over n2.  HZ: the
// inputs v[8..15] are zero and are not read (the zero-padded half of a
// Bluestein sequence).
template <bool HZ>
__device__ __forceinline__ void dft16(double2 *v)
{
    double2 a[4][4];
#pragma unroll
    for (int n2 = 0; n2 < 4; n2++)
    {
        if constexpr (HZ)
        {
            const double2 x0 = v[n2], x1 = v[4 + n2];
            a[n2][0] = add2(x0, x1);
            a[n2][1] = add2(x0, mul_mi(x1));
            a[n2][2] = sub2(x0, x1);
            a[n2][3] = sub2(x0, mul_mi(x1));
        }
        else
        {
            a[n2][0] = v[n2];
            a[n2][1] = v[4 + n2];
            a[n2][2] = v[8 + n2];
            a[n2][3] = v[12 + n2];
            dft4(a[n2][0], a[n2][1], a[n2][2], a[n2][3]);
        }
    }
    a[1][1] = cmul(a[1][1], make_double2(C16, -S16));
    a[1][2] = make_double2((a[1][2].x + a[1][2].y) * RSQRT2,
                           (a[1][2].y - a[1][2].x) * RSQRT2);
    a[1][3] = cmul(a[1][3], make_double2(S16, -C16));
    a[2][1] = make_double2((a[2][1].x + a[2][1].y) * RSQRT2,
                           (a[2][1].y - a[2][1].x) * RSQRT2);
    a[2][2] = mul_mi(a[2][2]);
    a[2][3] = make_double2((a[2][3].y - a[2][3].x) * RSQRT2,
                           -(a[2][3].x + a[2][3].y) * RSQRT2);
    a[3][1] = cmul(a[3][1], make_double2(S16, -C16));
    a[3][2] = make_double2((a[3][2].y - a[3][2].x) * RSQRT2,
                           -(a[3][2].x + a[3][2].y) * RSQRT2);
    a[3][3] = cmul(a[3][3], make_double2(-C16, S16));
#pragma unroll
    for (int k1 = 0; k1 < 4; k1++)
    {
        dft4(a[0][k1], a[1][k1], a[2][k1], a[3][k1]);
        v[k1] = a[0][k1];
        v[k1 + 4] = a[1][k1];
        v[k1 + 8] = a[2][k1];
        v[k1 + 12] = a[3][k1];
    }
}

// 9 = 3 x 3 (n = 3 n1 + n2, k = k1 + 3 k2), twiddles exp(-2 pi i n2 k1 / 9)
__device__ __forceinline__ void dft9(double2 *v)
{
    double2 a[3][3];
#pragma unroll
    for (int n2 = 0; n2 < 3; n2++)
    {
        a[n2][0] = v[n2];
        a[n2][1] = v[3 + n2];
        a[n2][2] = v[6 + n2];
        dft3(a[n2]);
    }
    a[1][1] = cmul(a[1][1], make_double2(C9A, -S9A));
    a[1][2] = cmul(a[1][2], make_double2(C9B, -S9B));
    a[2][1] = cmul(a[2][1], make_double2(C9B, -S9B));
    a[2][2] = cmul(a[2][2], make_double2(C9D, -S9D));
#pragma unroll
    for (int k1 = 0; k1 < 3; k1++)
    {
        double2 b[3] = {a[0][k1], a[1][k1], a[2][k1]};
        dft3(b);
        v[k1] = b[0];
        v[k1 + 3] = b[1];
        v[k1 + 6] = b[2];
    }
}

// 6 = 2 x 3 and 12 = 3 x 4 by the prime-factor map (no twiddles): inputs
// n = (3 n1 + 2 n2) mod 6 and (4 n1 + 3 n2) mod 12, outputs
// k = (3 k1 + 4 k2) mod 6 and (4 k1 + 9 k2) mod 12
__device__ __forceinline__ void dft6(double2 *v)
{
    double2 e[3] = {v[0], v[2], v[4]}, o[3] = {v[3], v[5], v[1]};
    dft3(e);
    dft3(o);
#pragma unroll
    for (int k2 = 0; k2 < 3; k2++)
    {
        v[(4 * k2) % 6] = add2(e[k2], o[k2]);
        v[(3 + 4 * k2) % 6] = sub2(e[k2], o[k2]);
    }
}

__device__ __forceinline__ void dft12(double2 *v)
{
    double2 a[3][4];
#pragma unroll
    for (int n1 = 0; n1 < 3; n1++)
    {
#pragma unroll
        for (int n2 = 0; n2 < 4; n2++)
            a[n1][n2] = v[(4 * n1 + 3 * n2) % 12];
        dft4(a[n1][0], a[n1][1], a[n1][2], a[n1][3]);
    }
#pragma unroll
    for (int k2 = 0; k2 < 4; k2++)
    {
        double2 b[3] = {a[0][k2], a[1][k2], a[2][k2]};
        dft3(b);
#pragma unroll
        for (int k1 = 0; k1 < 3; k1++)
            v[(4 * k1 + 9 * k2) % 12] = b[k1];
    }
}

// 18 = 2 x 9 by the prime-factor (Good-Thomas) map, no twiddles: input
// n = (9 n1 + 2 n2) mod 18, output k = (9 k1 + 10 k2) mod 18
__device__ __forceinline__ void dft18(double2 *v)
{
    double2 e[9], o[9];
#pragma unroll
    for (int n2 = 0; n2 < 9; n2++)
    {
        e[n2] = v[(2 * n2) % 18];
        o[n2] = v[(9 + 2 * n2) % 18];
    }
    dft9(e);
    dft9(o);
#pragma unroll
    for (int k2 = 0; k2 < 9; k2++)
    {
        v[(10 * k2) % 18] = add2(e[k2], o[k2]);
        v[(9 + 10 * k2) % 18] = sub2(e[k2], o[k2]);
    }
}

template <int R, bool HZ = false>
__device__ __forceinline__ void dft(double2 *v)
{
    if constexpr (R == 2)
        dft2(v);
    else if constexpr (R == 3)
        dft3(v);
    else if constexpr (R == 4)
        dft4(v[0], v[1], v[2], v[3]);
    else if constexpr (R == 6)
        dft6(v);
    else if constexpr (R == 8)
    {
        if constexpr (HZ)
        {
#pragma unroll
            for (int r = 4; r < 8; r++)
                v[r] = make_double2(0.0, 0.0);
        }
        dft8(v);
    }
    else if constexpr (R == 9)
        dft9(v);
    else if constexpr (R == 12)
        dft12(v);
    else if constexpr (R == 16)
        dft16<HZ>(v);
    else
    {
        static_assert(R == 18, "radix");
        dft18(v);
    }
}

// w[r] = w[1]^r for r = 2..R-1: w[2^a] = w[2^(a-1)]^2 and
// w[2^a + b] = w[2^a] w[b] (b < 2^a), at most log2 R + 1 products deep
constexpr int hibit(int r)
{
    int h = 1;
    while (2 * h <= r)
        h *= 2;
    return h;
}

template <int R>
__device__ __forceinline__ void twiddle_powers(double2 *w)
{
#pragma unroll
    for (int r = 2; r < R; r++)
    {
        if (r == hibit(r))
            w[r] = cmul(w[r / 2], w[r / 2]);
        else
            w[r] = cmul(w[hibit(r)], w[r - hibit(r)]);
    }
}

// Input of the first pass: element i of the sequence to transform.
struct SrcSmem
{
    const double2 *s;
    __device__ __forceinline__ double2 operator()(int i) const
    {
        return s[pidx(i)];
    }
};

// j div Ns and j mod Ns (one division by the run-time stride)
__device__ __forceinline__ void divmod_ns(int j, int Ns, int &q, int &k)
{
    k = j % Ns;
    q = (j - k) / Ns;
}

// One Stockham pass of radix R over s[0..M): butterfly j reads element
// j + r M/R (twiddled by exp(-2 pi i (j mod Ns) r / (Ns R))) and writes its
// R outputs to elements (j - j mod Ns) R + j mod Ns + r Ns.  The first pass
// (Ns = 1, no twiddles) reads through `src`; a non-null `bh` multiplies the
// stored outputs by bh and conjugates them.  Plans have 64 | M and start
// with two radix-8 passes, so M/R and every Ns > 1 are multiples of 8: the
// padded positions of a butterfly's elements are then a base plus a
// constant stride (r (M/R + M/8R) for loads, r (Ns + Ns/8) for stores, and
// r for the first pass's stores, whose bases are multiples of 8).
template <int R, int V, class Src>
__device__ __forceinline__ void stockham_pass(double2 *s,
                                              const double2 *__restrict__ tw,
                                              int M, int Ns, int tid, int T,
                                              bool first, const Src &src,
                                              const double2 *__restrict__ bh)
{
    constexpr int BPT = (V + R - 1) / R;
    const int nb = M / R;
    const int step = M / (Ns * R);
    const int ld_stride = nb + (nb >> 3);
    const int st_stride = (Ns == 1) ? 1 : Ns + (Ns >> 3);
    double2 v[BPT][R];
    if (first)
    {
#pragma unroll
        for (int c = 0; c < BPT; c++)
        {
            const int j = tid + c * T;
            if (j < nb)
            {
#pragma unroll
                for (int r = 0; r < R; r++)
                    v[c][r] = src(j + r * nb);
                dft<R>(v[c]);
            }
        }
    }
    else
    {
#pragma unroll
        for (int c = 0; c < BPT; c++)
        {
            const int j = tid + c * T;
            if (j < nb)
            {
                int q, k;
                divmod_ns(j, Ns, q, k);
                // one table twiddle per butterfly, its powers by products
                double2 wp[R];
                wp[1] = __ldg(&tw[k * step]);
                twiddle_powers<R>(wp);
                const int b = pidx(j);
                v[c][0] = s[b];
#pragma unroll
                for (int r = 1; r < R; r++)
                    v[c][r] = cmul(s[b + r * ld_stride], wp[r]);
                dft<R>(v[c]);
            }
        }
    }
    __syncthreads();
#pragma unroll
    for (int c = 0; c < BPT; c++)
    {
        const int j = tid + c * T;
        if (j < nb)
        {
            int q, k;
            divmod_ns(j, Ns, q, k);
            const int d = q * Ns * R + k;
            const int b = pidx(d);
            if (bh)
            {
#pragma unroll
                for (int r = 0; r < R; r++)
                    s[b + r * st_stride] =
                        conj2(cmul(v[c][r], __ldg(&bh[d + r * Ns])));
            }
            else
            {
#pragma unroll
                for (int r = 0; r < R; r++)
                    s[b + r * st_stride] = v[c][r];
            }
        }
    }
    __syncthreads();
}

// Forward FFT of length M = 8^n8 4^n4 2^n2 3^n3 (passes in that order) of
// the sequence src(0..M), result in s (natural order).  One loop per radix
// keeps every pass's registers separate.
template <int V, class Src>
__device__ __forceinline__ void fft_m(double2 *s,
                                      const double2 *__restrict__ tw, int M,
                                      int4 np, int tid, int T, const Src &src,
                                      const double2 *__restrict__ bh_last)
{
    const int last = np.x + np.y + np.z + np.w - 1;
    int Ns = 1, p = 0;
    for (int i = 0; i < np.x; i++, p++, Ns *= 8)
        stockham_pass<8, V>(s, tw, M, Ns, tid, T, p == 0, src,
                            p == last ? bh_last : nullptr);
    for (int i = 0; i < np.y; i++, p++, Ns *= 4)
        stockham_pass<4, V>(s, tw, M, Ns, tid, T, p == 0, src,
                            p == last ? bh_last : nullptr);
    for (int i = 0; i < np.z; i++, p++, Ns *= 2)
        stockham_pass<2, V>(s, tw, M, Ns, tid, T, p == 0, src,
                            p == last ? bh_last : nullptr);
    for (int i = 0; i < np.w; i++, p++, Ns *= 3)
        stockham_pass<3, V>(s, tw, M, Ns, tid, T, p == 0, src,
                            p == last ? bh_last : nullptr);
}

// ---- the same transform with the whole plan known at compile time ----
// Radices, strides, thread counts and butterfly ranges become constants, so
// the index arithmetic of every pass folds away, and the larger radices cut
// the number of barrier-separated passes through shared memory (4608 = 16 16
// 18: three passes instead of five).  The lengths are those that Bluestein's
// algorithm can ask of one CTA, 2^a 3^b with 6 <= a and at most 9216; 6144,
// which ends in radix 3, serves the clusters alone (one CTA runs that length,
// and the direct transforms, by the run-time plan).  The first radix is 16 or
// 8 (the zero half of a chirped sequence is skipped there), the last of the
// others even (the half-output passes), and every pass keeps M / R and the
// stride a multiple of 8 (the padded layout).
struct CtPlan
{
    int M, n, r[4];
    int T;   // threads per row
};

constexpr CtPlan CT_PLANS[] = {
    {64, 2, {8, 8, 0, 0}, 4},        {128, 2, {16, 8, 0, 0}, 8},
    {192, 3, {8, 3, 8, 0}, 12},      {256, 2, {16, 16, 0, 0}, 16},
    {384, 3, {16, 3, 8, 0}, 24},     {512, 3, {16, 4, 8, 0}, 32},
    {576, 3, {8, 9, 8, 0}, 36},      {768, 3, {16, 3, 16, 0}, 48},
    {1024, 3, {16, 8, 8, 0}, 64},    {1152, 3, {16, 4, 18, 0}, 72},
    {1536, 3, {16, 12, 8, 0}, 128},  {1728, 3, {8, 12, 18, 0}, 144},
    {2048, 3, {16, 16, 8, 0}, 128},  {2304, 3, {16, 9, 16, 0}, 144},
    {3072, 3, {16, 12, 16, 0}, 256}, {3456, 3, {16, 12, 18, 0}, 288},
    {4096, 3, {16, 16, 16, 0}, 256}, {4608, 3, {16, 16, 18, 0}, 288},
    {5184, 4, {8, 9, 12, 6}, 432},   {6144, 4, {16, 16, 8, 3}, 384},
    {6912, 4, {16, 9, 6, 8}, 432},   {8192, 4, {16, 16, 8, 4}, 512},
    {9216, 4, {16, 16, 9, 4}, 576}};

constexpr CtPlan ct_plan(int M)
{
    for (const CtPlan &p : CT_PLANS)
        if (p.M == M)
            return p;
    return CtPlan{};
}

constexpr int ct_npass(int M) { return ct_plan(M).n; }
constexpr int ct_radix(int M, int p) { return ct_plan(M).r[p]; }
constexpr int ct_threads(int M) { return ct_plan(M).T; }

// rows per CTA: short transforms share one, so that a CTA has two warps
constexpr int ct_rows(int M)
{
    return M > 0 && ct_threads(M) < 64 ? 64 / ct_threads(M) : 1;
}

constexpr int ct_ns(int M, int p)
{
    int ns = 1;
    for (int i = 0; i < p; i++)
        ns *= ct_radix(M, i);
    return ns;
}

// read-only load that stays after the barrier before it (a volatile asm is
// not moved across the barrier's), so the twiddles of later passes are
// not hoisted into registers ahead of time
__device__ __forceinline__ double2 ld_tw(const double2 *p)
{
    double2 v;
    asm volatile("ld.global.nc.v2.f64 {%0, %1}, [%2];"
                 : "=d"(v.x), "=d"(v.y)
                 : "l"(p));
    return v;
}

// HZ (first pass of a Bluestein sequence only): elements M/2.. are zero
// (M >= 2H), so a butterfly's upper R/2 inputs are neither read nor added.
// HO (last pass of Bluestein's second FFT only): outputs M/2.. are never
// read (H <= M/2), so they are neither computed nor stored.
template <int R, int M, int NS, bool FIRST, bool BH, bool HZ,
          bool HO = false, class Src>
__device__ __forceinline__ void stockham_ct(double2 *s,
                                            const double2 *__restrict__ tw,
                                            int tid, const Src &src,
                                            const double2 *__restrict__ bh)
{
    constexpr int T = ct_threads(M);
    constexpr int nb = M / R;
    constexpr int BPT = (nb + T - 1) / T;
    constexpr int step = M / (NS * R);
    constexpr int ld_stride = nb + (nb >> 3);
    static_assert(nb % 8 == 0 && (NS == 1 || NS % 8 == 0), "padding");
    static_assert(!FIRST || R % 8 == 0, "first pass radix");
    static_assert(!HZ || (FIRST && (R == 16 || R == 8)), "zero half");
    static_assert(!HO || (NS * R == M && R % 2 == 0 && !BH), "half output");
    // padded offset of a butterfly's output r from its first one: the
    // first pass writes R consecutive elements from a multiple of 8
    auto st_off = [](int r) {
        return NS == 1 ? r + (r >> 3) : r * (NS + (NS >> 3));
    };
    double2 v[BPT][R];
#pragma unroll
    for (int c = 0; c < BPT; c++)
    {
        const int j = tid + c * T;
        if (j < nb)
        {
            if constexpr (FIRST)
            {
#pragma unroll
                for (int r = 0; r < (HZ ? R / 2 : R); r++)
                    v[c][r] = src(j + r * nb);
            }
            else
            {
                const int k = j % NS;
                double2 wp[R];
                wp[1] = ld_tw(&tw[k * step]);
                twiddle_powers<R>(wp);
                const int b = pidx(j);
                v[c][0] = s[b];
#pragma unroll
                for (int r = 1; r < R; r++)
                    v[c][r] = cmul(s[b + r * ld_stride], wp[r]);
            }
            dft<R, HZ>(v[c]);
        }
    }
    __syncthreads();
#pragma unroll
    for (int c = 0; c < BPT; c++)
    {
        const int j = tid + c * T;
        if (j < nb)
        {
            const int k = j % NS;
            const int d = (j / NS) * NS * R + k;
            const int b = pidx(d);
            if constexpr (BH)
            {
#pragma unroll
                for (int r = 0; r < R; r++)
                    s[b + st_off(r)] =
                        conj2(cmul(v[c][r], ld_tw(&bh[d + r * NS])));
            }
            else
            {
#pragma unroll
                for (int r = 0; r < (HO ? R / 2 : R); r++)
                    s[b + st_off(r)] = v[c][r];
            }
        }
    }
    __syncthreads();
}

// passes P..PEND-1 of FFT_M (compile-time plan); the FFT's last pass
// multiplies by bh when given; HZ: the upper half of the input sequence
// is zero; HO: only the lower half of the output is wanted
template <int M, int P, bool HZ, int PEND = ct_npass(M), bool HO = false,
          class Src>
__device__ __forceinline__ void fft_ct(double2 *s,
                                       const double2 *__restrict__ tw, int tid,
                                       const Src &src,
                                       const double2 *__restrict__ bh_last)
{
    if constexpr (P < PEND)
    {
        constexpr int R = ct_radix(M, P);
        constexpr int NS = ct_ns(M, P);
        constexpr bool Z = HZ && P == 0;
        if constexpr (P == ct_npass(M) - 1)
        {
            if (bh_last)
                stockham_ct<R, M, NS, P == 0, true, Z>(s, tw, tid, src,
                                                          bh_last);
            else
                stockham_ct<R, M, NS, P == 0, false, Z, HO>(
                    s, tw, tid, src, nullptr);
        }
        else
            stockham_ct<R, M, NS, P == 0, false, Z>(s, tw, tid, src,
                                                       nullptr);
        fft_ct<M, P + 1, HZ, PEND, HO>(s, tw, tid, src, bh_last);
    }
}

// The last pass of the second FFT_M of Bluestein's algorithm (compile-time
// plan, even last radix) handed straight to its consumer: output
// k = j + r M/R of butterfly j goes to out(k, value) for k < H <= M/2.
// Nothing is stored in shared memory, so the pass needs no barrier.
template <int M, class Out>
__device__ __forceinline__ void fft_ct_last_out(const double2 *s,
                                                const double2 *__restrict__ tw,
                                                int tid, int H, const Out &out)
{
    constexpr int P = ct_npass(M) - 1;
    constexpr int R = ct_radix(M, P);
    constexpr int NS = ct_ns(M, P);
    static_assert(NS * R == M && R % 2 == 0, "last pass");
    constexpr int T = ct_threads(M);
    constexpr int BPT = (NS + T - 1) / T;
    constexpr int ld_stride = NS + (NS >> 3);
#pragma unroll 1
    for (int c = 0; c < BPT; c++)
    {
        const int j = tid + c * T;
        if (j < NS)
        {
            double2 wp[R], v[R];
            wp[1] = ld_tw(&tw[j]);
            twiddle_powers<R>(wp);
            const int b = pidx(j);
            v[0] = s[b];
#pragma unroll
            for (int r = 1; r < R; r++)
                v[r] = cmul(s[b + r * ld_stride], wp[r]);
            dft<R>(v);
            // H <= M/2: the outputs of the upper half are never used
#pragma unroll
            for (int r = 0; r < R / 2; r++)
                if (j + r * NS < H)
                    out(j + r * NS, v[r]);
        }
    }
}

// Complex DFT of length H of the sequence z(0..H), zero-padded to M when
// Bluestein is used; `pre` returns z_j already multiplied by the chirp
// (Bluestein) and 0 for j >= H.  On return the DFT value k is dft_h_out(k).
template <int V, int MC, class Pre>
__device__ __forceinline__ void dft_h(double2 *s, const RfftArgs &A, int tid,
                                      int T, const Pre &pre)
{
    if constexpr (MC > 0)
    {
        // plan fixed at compile time (A.M == MC, Bluestein)
        fft_ct<MC, 0, true>(s, A.tw, tid, pre, A.bh);
        fft_ct<MC, 0, false, ct_npass(MC), true>(s, A.tw, tid, SrcSmem{s},
                                                    nullptr);
    }
    else
    {
        if (A.direct)
        {
            fft_m<V>(s, A.tw, A.M, A.npass, tid, T, pre, nullptr);
            return;
        }
        fft_m<V>(s, A.tw, A.M, A.npass, tid, T, pre, A.bh);
        fft_m<V>(s, A.tw, A.M, A.npass, tid, T, SrcSmem{s}, nullptr);
    }
}

// value k (< H) of the length-H DFT after dft_h
__device__ __forceinline__ double2 dft_h_out(const double2 *s,
                                             const RfftArgs &A, int k)
{
    if (A.direct)
        return s[pidx(k)];
    return cmul(__ldg(&A.w[k]), conj2(s[pidx(k)]));
}

// Analysis input: z_j = x_2j + i x_2j+1 times the chirp.
struct SrcRow
{
    const double2 *x2;
    const double2 *w;
    int H;
    __device__ __forceinline__ double2 operator()(int i) const
    {
        if (i >= H)
            return make_double2(0.0, 0.0);
        double2 z = x2[i];
        return w ? cmul(z, __ldg(&w[i])) : z;
    }
};

// Analysis input from float rows (the single-precision mode)
struct SrcRowF
{
    const float2 *x2;
    const double2 *w;
    int H;
    __device__ __forceinline__ double2 operator()(int i) const
    {
        if (i >= H)
            return make_double2(0.0, 0.0);
        const float2 f = x2[i];
        double2 z = make_double2((double)f.x, (double)f.y);
        return w ? cmul(z, __ldg(&w[i])) : z;
    }
};

// Synthesis input: conj Z_k times the chirp, with
// Z_k = (X_k + conj X_H-k) + i e^(i pi k/H) (X_k - conj X_H-k) and X_k = 0
// above kmax (the inverse DFT is conj(DFT(conj Z))).
struct SrcSpectrum
{
    const double2 *X;
    const double2 *w;
    const double2 *ht;
    int H, kmax;
    __device__ __forceinline__ double2 operator()(int k) const
    {
        if (k >= H)
            return make_double2(0.0, 0.0);
        const int kh = H - k;
        double2 xk = k <= kmax ? X[k] : make_double2(0.0, 0.0);
        double2 xh = kh <= kmax ? conj2(X[kh]) : make_double2(0.0, 0.0);
        double2 e = cmul(conj2(__ldg(&ht[k])), sub2(xk, xh));
        double2 zc = make_double2(xk.x + xh.x - e.y, -(xk.y + xh.y + e.x));
        return w ? cmul(zc, __ldg(&w[k])) : zc;
    }
};

// Synthesis input of the quarter-length transform.  A row of length 4H
// whose spectrum X stops below H gives, with a = X_k, b = conj X_H-k and
// o = exp(2 pi i k / 4H),
//   V_0[k] = (a + b) + i o (a - i b),
//   V_1[k] = o^2 (a - b) + i o^3 (a + i b),
// and the inverse DFT of length H of V_rho holds the pairs
// (x_4q+2rho, x_4q+2rho+1) of the row (the four residues of the row index
// mod 4, paired into two complex sequences).  Returns conj V_rho[k] times
// the chirp, as SrcSpectrum.
struct SrcQuarter
{
    const double2 *X;
    const double2 *w;
    const double2 *w4;
    int H, kmax, rho;
    __device__ __forceinline__ double2 operator()(int k) const
    {
        if (k >= H)
            return make_double2(0.0, 0.0);
        const int kh = H - k;
        const double2 a = k <= kmax ? X[k] : make_double2(0.0, 0.0);
        const double2 b =
            (k >= 1 && kh <= kmax) ? conj2(X[kh]) : make_double2(0.0, 0.0);
        const double2 o = __ldg(&w4[k]);
        double2 v;
        if (rho == 0)
        {
            const double2 t = cmul(o, add2(a, mul_mi(b)));
            v = make_double2(a.x + b.x - t.y, a.y + b.y + t.x);
        }
        else
        {
            const double2 o2 = cmul(o, o);
            const double2 o3 = cmul(o2, o);
            const double2 u = cmul(o2, sub2(a, b));
            const double2 t = cmul(o3, sub2(a, mul_mi(b)));
            v = make_double2(u.x - t.y, u.y + t.x);
        }
        return cmul(conj2(v), __ldg(&w[k]));
    }
};

// Bluestein kernel b_n = conj w_|n| on the circle of length M
struct SrcKernel
{
    const double2 *w;
    int H, M;
    __device__ __forceinline__ double2 operator()(int n) const
    {
        if (n < H)
            return conj2(w[n]);
        if (n > M - H)
            return conj2(w[M - n]);
        return make_double2(0.0, 0.0);
    }
};

// Synthesis input of a row of odd length L: the Hermitian extension Y of
// the spectrum (Y_k = X_k for k <= (L - 1)/2, conj X_L-k above, zero above
// kmax, the imaginary part of X_0 ignored), conjugated and chirped; the row
// is the real part of the inverse DFT of length H = L.
struct SrcSpectrumOdd
{
    const double2 *X;
    const double2 *w;
    int H, kmax;
    __device__ __forceinline__ double2 operator()(int k) const
    {
        if (k >= H)
            return make_double2(0.0, 0.0);
        double2 y = make_double2(0.0, 0.0);
        if (2 * k < H)
        {
            if (k <= kmax)
                y = X[k];
            if (k == 0)
                y.y = 0.0;
        }
        else if (H - k <= kmax)
            y = conj2(X[H - k]);
        return cmul(conj2(y), __ldg(&w[k]));
    }
};

// ---- transforms longer than one CTA's shared memory ----
// A cluster of C CTAs owns a row; CTA q holds Mc = M / C values.  FFT_M of
// a sequence a is computed as
//   y_q[i] = w_M^(i q) sum_k a[i + k Mc] w_C^(k q)    (radix-C decimation
//            in frequency across the CTAs, folded into the loads of the
//            first local pass), then FFT_Mc(y_q)[l] = FFT_M(a)[C l + q],
// so every CTA holds one residue class of the spectrum, in which the
// pointwise product of Bluestein's algorithm needs no exchange.  The second
// FFT_M takes its input by residue classes (decimation in time): each CTA
// transforms its class, U_q = FFT_Mc, and
//   v_t = sum_q w_M^(q t) U_q[t mod Mc]
// is gathered through distributed shared memory for the outputs t a CTA
// writes.

// Input of the first local pass of CTA q: a = src(0..M) vanishes from nz
// on, so blocks k with k Mc >= nz are not read.
template <class Src>
struct SrcClusterDif
{
    Src src;
    const double2 *twM;
    int q, C, Mc, M, nz;
    __device__ __forceinline__ double2 operator()(int i) const
    {
        // i < Mc and q < C, C a power of two: k q mod C is a mask and
        // i q < Mc C = M needs no reduction
        double2 acc = src(i);
        for (int k = 1; k < C && k * Mc < nz; k++)
        {
            const int kq = (k * q) & (C - 1);
            acc = add2(acc, cmul(src(i + k * Mc), __ldg(&twM[kq * Mc])));
        }
        if (q == 0)
            return acc;
        return cmul(acc, __ldg(&twM[i * q]));
    }
};

// v_t of the second FFT_M (t < M) from the residue transforms U_q held in
// the shared memory of the cluster's CTAs.
__device__ __forceinline__ double2 cluster_v(
    const cooperative_groups::cluster_group &cl, double2 *s,
    const double2 *__restrict__ twM, int C, int Mc, int M, int t)
{
    const int pj = pidx(t % Mc);
    double2 acc = *cl.map_shared_rank(s + pj, 0);
    // e = qq t mod M by repeated addition (t < M)
    int e = 0;
    for (int qq = 1; qq < C; qq++)
    {
        e += t;
        if (e >= M)
            e -= M;
        const double2 u = *cl.map_shared_rank(s + pj, qq);
        acc = add2(acc, cmul(u, __ldg(&twM[e])));
    }
    return acc;
}

} // namespace

// Register cap NR: M / 16 <= 576 threads of 96 registers with V = 16 values
// per thread (five warps on one scheduler's 16384 registers; two CTAs of
// 288 threads per SM up to M = 4608).
constexpr int RFFT_NR = 96;
#define RFFT_BOUNDS(NR) __maxnreg__(NR)

// This CTA's part of a launch: rows of one batch entry (blockIdx.y), or of A
// itself.  BATCH = false compiles the former out: with it the run-time plans
// spill 520 bytes a thread (rows of GL nmax 767 23 us in the place of 19, of
// nmax 1151 56 in the place of 47, 90 rows of 3001 points 43 in the place of
// 37), so a launch without a batch has kernels of its own there.
template <bool BATCH>
__device__ __forceinline__ RfftRows pick_rows(const RfftArgs &A)
{
    if constexpr (BATCH)
        if (A.batch)
            return A.batch[blockIdx.y];
    return {A.x, A.X, A.kmax};
}

// Analysis direction: real rows x[row][0..L) -> X[row][0..kmax]; one CTA
// per ct_rows(MC) rows (a loop over rows would let the compiler hoist every
// pass's twiddles out of it and run out of registers).
template <bool F32, int MC>
__global__ void RFFT_BOUNDS(RFFT_NR) k_rfft_fwd(RfftArgs A)
{
    extern __shared__ __align__(16) double2 smem[];
    constexpr int RP = ct_rows(MC);
    const int T = MC > 0 ? ct_threads(MC) : (int)blockDim.x;
    const int sub = RP > 1 ? (int)threadIdx.x / T : 0;
    const int tid = (int)threadIdx.x - sub * T;
    double2 *s = smem + sub * (MC + MC / 8);
    const int H = A.H;
    // rows beyond the last are transformed again and not stored
    long long row = (long long)blockIdx.x * RP + sub;
    const bool mine = RP == 1 || row < A.nrows;
    if (!mine)
        row = A.nrows - 1;
    if constexpr (F32)
    {
        const float *xf = reinterpret_cast<const float *>(A.x);
        SrcRowF src{reinterpret_cast<const float2 *>(xf + row * A.ldx),
                    A.direct ? nullptr : A.w, H};
        dft_h<16, MC>(s, A, tid, T, src);
    }
    else
    {
        SrcRow src{reinterpret_cast<const double2 *>(A.x + row * A.ldx),
                   A.direct ? nullptr : A.w, H};
        dft_h<16, MC>(s, A, tid, T, src);
    }
    if (!mine)
        return;
    double2 *X = A.X + row * A.ldX;
    for (int k = tid; k <= A.kmax; k += T)
    {
        const int ka = (k == H) ? 0 : k;
        const int kb = (k == 0) ? 0 : H - k;
        double2 zk = dft_h_out(s, A, ka);
        double2 zh = conj2(dft_h_out(s, A, kb));
        double2 e = cmul(__ldg(&A.ht[k]), sub2(zk, zh));
        double2 sm = add2(zk, zh);
        X[k] = make_double2(0.5 * (sm.x + e.y), 0.5 * (sm.y - e.x));
    }
}

// Synthesis direction: X[row][0..kmax] (zero above) -> real rows x[row].
// Output of the synthesis direction: x_2k + i x_2k+1 = conj of DFT value
// k, which Bluestein's algorithm gives as w_k conj(second FFT output k).
template <bool F32>
struct OutRow
{
    void *x2;
    const double2 *w;
    __device__ __forceinline__ void operator()(int k, double2 v) const
    {
        const double2 z = cmul(__ldg(&w[k]), conj2(v));
        if constexpr (F32)
            reinterpret_cast<float2 *>(x2)[k] =
                make_float2((float)z.x, (float)-z.y);
        else
            reinterpret_cast<double2 *>(x2)[k] = conj2(z);
    }
};

template <bool F32, int MC, bool BATCH = true>
__global__ void RFFT_BOUNDS(RFFT_NR) k_rfft_inv(RfftArgs A)
{
    extern __shared__ __align__(16) double2 smem[];
    constexpr int RP = ct_rows(MC);
    const int T = MC > 0 ? ct_threads(MC) : (int)blockDim.x;
    const int sub = RP > 1 ? (int)threadIdx.x / T : 0;
    const int tid = (int)threadIdx.x - sub * T;
    double2 *s = smem + sub * (MC + MC / 8);
    const RfftRows R = pick_rows<BATCH>(A);
    long long row = (long long)blockIdx.x * RP + sub;
    const bool mine = RP == 1 || row < A.nrows;
    if (!mine)
        row = A.nrows - 1;
    SrcSpectrum src{R.X + row * A.ldX, A.direct ? nullptr : A.w, A.ht, A.H,
                    R.kmax};
    if constexpr (MC > 0)
    {
        // Bluestein with the second FFT's last pass writing the row
        void *x2 = F32 ? (void *)(reinterpret_cast<float *>(R.x) +
                                  row * A.ldx)
                       : (void *)(R.x + row * A.ldx);
        fft_ct<MC, 0, true>(s, A.tw, tid, src, A.bh);
        fft_ct<MC, 0, false, ct_npass(MC) - 1>(s, A.tw, tid, SrcSmem{s},
                                               nullptr);
        fft_ct_last_out<MC>(s, A.tw, tid, mine ? A.H : 0,
                            OutRow<F32>{x2, A.w});
    }
    else
    {
        dft_h<16, 0>(s, A, tid, T, src);
        if constexpr (F32)
        {
            float *xf = reinterpret_cast<float *>(R.x);
            float2 *x2 = reinterpret_cast<float2 *>(xf + row * A.ldx);
            for (int j = tid; j < A.H; j += T)
            {
                const double2 z = conj2(dft_h_out(s, A, j));
                x2[j] = make_float2((float)z.x, (float)z.y);
            }
        }
        else
        {
            double2 *x2 = reinterpret_cast<double2 *>(R.x + row * A.ldx);
            for (int j = tid; j < A.H; j += T)
                x2[j] = conj2(dft_h_out(s, A, j));
        }
    }
}

// launch of the one-CTA kernels with the compile-time plan MC
template <int MC>
static cudaError_t rfft_ct_launch(const RfftArgs &A, bool inverse,
                                  cudaStream_t st)
{
    constexpr int RP = ct_rows(MC);
    constexpr int T = ct_threads(MC) * RP;
    constexpr size_t smem = (size_t)RP * (MC + MC / 8) * sizeof(double2);
    const dim3 grid((unsigned)((A.nrows + RP - 1) / RP),
                    A.batch ? (unsigned)A.nbatch : 1u);
    void (*const fn)(RfftArgs) =
        A.f32_rows ? (inverse ? k_rfft_inv<true, MC> : k_rfft_fwd<true, MC>)
                   : (inverse ? k_rfft_inv<false, MC> : k_rfft_fwd<false, MC>);
    if constexpr (smem > 48 * 1024)
    {
        // beyond the default limit; once per kernel
        static const cudaError_t attr = [] {
            const void *f[] = {(const void *)k_rfft_inv<true, MC>,
                               (const void *)k_rfft_fwd<true, MC>,
                               (const void *)k_rfft_inv<false, MC>,
                               (const void *)k_rfft_fwd<false, MC>};
            for (const void *p : f)
            {
                const cudaError_t e = cudaFuncSetAttribute(
                    p, cudaFuncAttributeMaxDynamicSharedMemorySize,
                    (int)smem);
                if (e != cudaSuccess)
                    return e;
            }
            return cudaSuccess;
        }();
        if (attr != cudaSuccess)
            return attr;
    }
    fn<<<grid, T, smem, st>>>(A);
    return cudaGetLastError();
}

} // namespace cb
