// Tables of the two-degree recurrence (two.cuh), the latitudes of a grid in
// the form its kernels read, and the passes that take coefficients into and
// out of its normalisation.
#include <cstdint>

#include "common.cuh"
#include "kernels.h"
#include "two.cuh"

namespace cb
{

namespace
{

// eps_n^2 of order m at n = m + i, in double-double (the products are exact
// integers below 2^53)
__device__ __forceinline__ dd eps2(long long m, long long i)
{
    const double num = (double)i * (double)(2 * m + i);
    const double n = (double)(m + i);
    return dd_div(dd{num, 0.0}, dd{4.0 * n * n - 1.0, 0.0});
}

// k_l+1^2 / k_l-1^2
__device__ __forceinline__ dd k_ratio(long long m, long long l)
{
    const double i = 2.0 * (double)l, d = (double)(2 * m), n = i + (double)m;
    // (eps_i+1 eps_i)^2 / (eps_i+2 eps_i+3)^2, each factor exact
    dd num = dd_mul(dd{(i + 1.0) * (d + i + 1.0), 0.0}, dd{i * (d + i), 0.0});
    num = dd_mul(num, dd_mul(dd{4.0 * (n + 2.0) * (n + 2.0) - 1.0, 0.0},
                             dd{4.0 * (n + 3.0) * (n + 3.0) - 1.0, 0.0}));
    dd den = dd_mul(dd{(i + 2.0) * (d + i + 2.0), 0.0},
                    dd{(i + 3.0) * (d + i + 3.0), 0.0});
    den = dd_mul(den, dd_mul(dd{4.0 * n * n - 1.0, 0.0},
                             dd{4.0 * (n + 1.0) * (n + 1.0) - 1.0, 0.0}));
    return dd_div(num, den);
}

constexpr int TAB_THREADS = 128;

} // namespace

// One block per order.  k_l^2 is a product of k_ratio over every second l
// (two interleaved chains from k_0, k_1): each thread multiplies a
// contiguous stretch of l, the block scans the stretches, and the second
// walk writes
//     ab = (alpha_l, beta_l),  ag = (alpha_l, gamma_l),
//     kw = (k_l eps_m+2l+1, k_l eps_m+2l+2, k_l),
// and sm[m] = S_m = P_mm / cos^m.
// k_0 = 1 / eps_m+1, so s_0 = P_mm; k_1 = k_0 sqrt(k_ratio(1)) rounded (any
// value serves; this one keeps the two chains level).
__global__ void k_two_tables(long long nmax, const double *sg, double2 *ab,
                             double2 *ag, double *kw, double *sm, long long TL)
{
    if (threadIdx.x == 0)
        sm[blockIdx.x] = scalbn(sg[2 * blockIdx.x],
                                -(int)sg[2 * blockIdx.x + 1]);
    __shared__ dd chain[2][TAB_THREADS];
    const long long m = blockIdx.x;
    const long long nl = two_len(nmax, m);
    const long long c0 = two_col0(nmax, m);
    const int tid = threadIdx.x;
    // even stretches keep the parity of l fixed per slot
    const long long len = 2 * ((nl + 1 + 2 * TAB_THREADS - 1) /
                               (2 * TAB_THREADS));
    const long long l0 = tid * len;
    // k^2 of l0 and l0 + 1 relative to k^2 of 0 and 1: the products over the
    // stretches before this one
    dd p0{1.0, 0.0}, p1{1.0, 0.0};
    for (long long l = l0; l < l0 + len && l <= nl; l += 2)
    {
        p0 = dd_mul(p0, k_ratio(m, l + 1));   // k_l+2 / k_l
        p1 = dd_mul(p1, k_ratio(m, l + 2));   // k_l+3 / k_l+1
    }
    chain[0][tid] = p0;
    chain[1][tid] = p1;
    __syncthreads();
    for (int off = 1; off < TAB_THREADS; off <<= 1)
    {
        dd a0{1.0, 0.0}, a1{1.0, 0.0};
        if (tid >= off)
        {
            a0 = chain[0][tid - off];
            a1 = chain[1][tid - off];
        }
        __syncthreads();
        if (tid >= off)
        {
            chain[0][tid] = dd_mul(a0, chain[0][tid]);
            chain[1][tid] = dd_mul(a1, chain[1][tid]);
        }
        __syncthreads();
    }
    const dd k0sq = dd_div(dd{1.0, 0.0}, eps2(m, 1));
    const double r1 = sqrt(k_ratio(m, 1).hi);
    dd ke = k0sq, ko = dd_mul(k0sq, dd{r1, 0.0});
    if (tid > 0)
    {
        ke = dd_mul(ke, chain[0][tid - 1]);
        ko = dd_mul(ko, chain[1][tid - 1]);
    }
    for (long long l = l0; l < l0 + len && l < nl; l += 2)
    {
        // k_l^2 = ke, k_l+1^2 = ko, k_l+2^2
        const dd kn = dd_mul(ke, k_ratio(m, l + 1));
        dd ks[3] = {ke, ko, kn};
#pragma unroll
        for (int h = 0; h < 2; h++)
        {
            const long long ll = l + h;
            if (ll >= nl)
                break;
            const dd e1 = eps2(m, 2 * ll + 1), e2 = eps2(m, 2 * ll + 2),
                     e3 = eps2(m, 2 * ll + 3);
            const dd alpha = dd_sqrt(
                dd_div(ks[h], dd_mul(ks[h + 1], dd_mul(e2, e3))));
            const dd A = dd_add(e1, e2);
            const dd beta = dd_neg(dd_mul(A, alpha));
            const dd gamma = dd_add(alpha, beta);
            ab[c0 + ll] = make_double2(alpha.hi, beta.hi);
            ag[c0 + ll] = make_double2(alpha.hi, gamma.hi);
            kw[c0 + ll] = dd_sqrt(dd_mul(ks[h], e1)).hi;
            kw[TL + c0 + ll] = dd_sqrt(dd_mul(ks[h], e2)).hi;
            kw[2 * TL + c0 + ll] = dd_sqrt(ks[h]).hi;
        }
        const dd kon = dd_mul(ko, k_ratio(m, l + 2));
        ke = kn;
        ko = kon;
    }
}

// ---------------------------------------------------------------------------
// Latitudes.  Per pair, from the double-double sine and cosine of its
// latitude (Taylor series of lat / 8, doubled three times): t, u rounded;
// z = x2, or -u2 for the pairs below `polar`; and (by > 0) the power
// table of two_seed, POW_STRETCH entries per thread.  The first row of blocks
// also copies the call's page-locked staging to the device (one launch in the
// place of a copy and a memset), clears its counters and fills the powers
// rhop[n] = rho^n, n = 0..nmax, of the one radius ratio rho (1 + drho)
// of the call (drho: its relative rounding error).  Latency-bound: chains
// of some hundred dependent operations whatever the sizes (with the series
// by nested double-double divisions the kernel took 13 us).
// ---------------------------------------------------------------------------
namespace
{

constexpr int POW_STRETCH = 8;
constexpr int GEO_THREADS = 128;

__host__ __device__ __forceinline__ int geo_blocks_x(const GeometryArgs &G)
{
    // a thread per pair, and per 16 bytes of the staging: each of its reads
    // takes more than a microsecond, so none waits for another
    const long long n = G.words / 2 > G.npairs ? G.words / 2 : G.npairs;
    return n > 0 ? (int)((n + GEO_THREADS - 1) / GEO_THREADS) : 1;
}

__host__ __device__ __forceinline__ int geo_blocks_y(const GeometryArgs &G)
{
    return 1 + (G.npow + POW_STRETCH - 1) / POW_STRETCH;
}

// (mantissa, exponent) of a dd, the mantissa in [1, 2)
struct ddx
{
    dd v;
    int e;
};

__device__ __forceinline__ ddx ddx_norm(dd v, int e)
{
    const int h = ((__double2hiint(v.hi) >> 20) & 0x7ff) - 1023;
    if (h == -1023)
        return {dd{0.0, 0.0}, 0};
    const double f = pow2i(-h);
    return {dd{v.hi * f, v.lo * f}, e + h};
}

__device__ __forceinline__ ddx ddx_mul(ddx a, ddx b)
{
    return ddx_norm(dd_mul(a.v, b.v), a.e + b.e);
}

__device__ ddx ddx_pow(ddx b, long long k)
{
    ddx r{dd{1.0, 0.0}, 0};
    while (k)
    {
        if (k & 1)
            r = ddx_mul(r, b);
        k >>= 1;
        if (k)
            b = ddx_mul(b, b);
    }
    return r;
}

} // namespace

__device__ void geometry_block(const GeometryArgs &G, int bx, int by)
{
    const int p = bx * GEO_THREADS + (int)threadIdx.x;
    if (by == 0)
    {
        if (bx == 0 && threadIdx.x < GEO_CLEAR_WORDS)
            G.clear[threadIdx.x] = 0u;
        // (an even number of words)
        if (2LL * p < G.words)
            reinterpret_cast<double2 *>(G.dst)[p] =
                reinterpret_cast<const double2 *>(G.src)[p];
        if (G.rhop)
            for (long long n = p; n <= G.nmax;
                 n += (long long)geo_blocks_x(G) * GEO_THREADS)
            {
                const ddx v = ddx_pow(
                    ddx_norm(dd_fast(G.rho, G.rho * G.drho), 0), n);
                G.rhop[n] = scalbn(v.v.hi, v.e);
            }
    }
    if (p >= G.npairs || G.plain)
        return;
    // sin h / h and cos h at h = lat / 8 (h^2 < 0.04): the terms from h^6 on
    // in double (below 2^-26, so good to 2^-79), the first two in
    // double-double; 1/6, 1/120, 1/2, 1/24 as sums of two doubles
    const double h = 0.125 * G.lat[p];
    const dd h2 = dd_mul(dd{h, 0.0}, dd{h, 0.0});
    const double w = h2.hi;
    const double ts =
        fma(w, fma(w, fma(w, fma(w, fma(w, -1.0 / 1307674368000.0,
                                        1.0 / 6227020800.0),
                                 -1.0 / 39916800.0),
                          1.0 / 362880.0),
                   -1.0 / 5040.0),
            0.0);
    const double tc =
        fma(w, fma(w, fma(w, fma(w, fma(w, -1.0 / 87178291200.0,
                                        1.0 / 479001600.0),
                                 -1.0 / 3628800.0),
                          1.0 / 40320.0),
                   -1.0 / 720.0),
            0.0);
    const dd one{1.0, 0.0};
    dd s = dd_add(dd{1.0 / 120.0, 0x1.1111111111111p-63}, dd{ts, 0.0});
    dd c = dd_add(dd{1.0 / 24.0, 0x1.5555555555555p-59}, dd{tc, 0.0});
    s = dd_add(dd{-1.0 / 6.0, -0x1.5555555555555p-57}, dd_mul(h2, s));
    c = dd_add(dd{-0.5, 0.0}, dd_mul(h2, c));
    s = dd_add(one, dd_mul(h2, s));
    c = dd_add(one, dd_mul(h2, c));
    s = dd_mul(s, dd{h, 0.0});
    for (int j = 0; j < 3; j++)
    {
        const dd s2 = dd_mul(s, s);
        s = dd_mul(s, c);
        s = dd{2.0 * s.hi, 2.0 * s.lo};
        c = dd_add(one, dd{-2.0 * s2.hi, -2.0 * s2.lo});
    }
    if (by == 0)
    {
        const bool given = p < G.given;
        G.t[p] = given ? G.src[4 * (long long)G.npairs + p] : s.hi;
        G.u[p] = given ? G.src[5 * (long long)G.npairs + p] : c.hi;
        G.z[p] = p < G.polar ? -dd_mul(c, c).hi : dd_mul(s, s).hi;
        return;
    }
    const int e0 = (by - 1) * POW_STRETCH;
    const int e1 = min(e0 + POW_STRETCH, G.npow);
    const ddx u = ddx_norm(c, 0);
    // the first POW_LOW entries u^e, then u^(POW_LOW j)
    ddx step = u, v;
    if (e0 < POW_LOW)
        v = ddx_pow(u, e0);
    else
    {
        step = ddx_pow(u, POW_LOW);
        v = ddx_pow(step, e0 - POW_LOW);
    }
    for (int e = e0; e < e1; e++)
    {
        G.pw[(size_t)e * G.npairs + p] = make_double2(v.v.hi, (double)v.e);
        v = ddx_mul(v, step);
    }
}

__global__ void k_geometry(GeometryArgs G)
{
    geometry_block(G, (int)blockIdx.x, (int)blockIdx.y);
}

// ---------------------------------------------------------------------------
// Coefficients of one set in the recurrences' normalisations.  For every
// (order, l) the two-degree pairs
//     (k_l (eps C_m+2l + eps C_m+2l+2), the same of S),  (k_l C_m+2l+1, ..),
// and, with cs not null, the one-degree (ct C, ct S) (leg.cuh), of every
// family of shs_two.cu that A asks for in the place of C, S (the two-degree
// pairs of G and J as the differences described there).  Degrees above
// nmax and S_n0 count as zero; rhop (or null) multiplies degree n first, dr
// the factors of a radial derivative.
// Layouts of the degree-ntab tables.  Memory-bound, one pass.  The first
// `geo` blocks are k_geometry's (which a call without rhop does not have to
// wait for): one launch and its latency less.
// ---------------------------------------------------------------------------
__global__ void k_two_scale(ScaleArgs A, long long m_lo, GeometryArgs G,
                            int geo)
{
    if ((int)blockIdx.x < geo)
    {
        const int nx = geo_blocks_x(G);
        geometry_block(G, (int)blockIdx.x % nx, (int)blockIdx.x / nx);
        return;
    }
    const long long m = m_lo + blockIdx.x - geo;
    const long long nmax = A.nmax;
    if (m > nmax)
        return;
    const long long c0 = two_col0(A.ntab, m);
    const long long t0 = tri_col0(A.ntab, m) - m;
    if (!A.cs2)
    {
        // the one-degree form of C, S alone
        const long long s1 = tri_col0(A.shc_nmax, m) - m;
        for (long long n = m + threadIdx.x; n <= nmax; n += blockDim.x)
        {
            double k = A.tc[t0 + n];
            double vc = A.c[s1 + n], vs = m == 0 ? 0.0 : A.s[s1 + n];
            if (A.rhop)
            {
                vc *= A.rhop[n];
                vs *= A.rhop[n];
            }
            A.cs[t0 + n] = make_double2(k * vc, k * vs);
        }
        return;
    }
    const long long s0 = tri_col0(A.shc_nmax, m) - m;
    const long long nl = two_len(nmax, m);
    const long long TL = two_sum(A.ntab);
    const long long T1 = tri_size(A.ntab);
    // the degree's factor: radius ratio and radial derivative
    auto get = [&](long long n) {
        if (n > nmax)
            return make_double2(0.0, 0.0);
        double w = A.rhop ? A.rhop[n] : 1.0;
        if (A.dr >= 1)
            w *= (double)(n + 1);
        if (A.dr >= 2)
            w *= (double)(n + 2);
        return make_double2(w * A.c[s0 + n], m == 0 ? 0.0 : w * A.s[s0 + n]);
    };
    auto times = [](double w, double2 v) {
        return make_double2(w * v.x, w * v.y);
    };
    // member n of family f from the coefficients of degrees n and n + 1
    auto member = [&](int f, long long n, double2 v, double2 next) {
        const double nd = (double)n;
        switch (f)
        {
        case 0: return v;
        case 1: return times(nd, v);
        case 2: return times(nd * (nd + 1.0), v);
        default:
        {
            // e_n+1: cos(lat) dP_n+1 = e_n+1 P_n - (n + 1) t P_n+1
            const double q = nd + 1.0, md = (double)m;
            const double e = sqrt((q - md) * (q + md) * (2.0 * q + 1.0) /
                                  (2.0 * q - 1.0));
            return times(f == 3 ? e : e * (q + 1.0), next);
        }
        }
    };
    for (long long l = threadIdx.x; l < nl; l += blockDim.x)
    {
        const long long n = m + 2 * l;
        const double2 v0 = get(n), v1 = get(n + 1), v2 = get(n + 2);
        const double2 v3 = A.nfam > 1 ? get(n + 3) : v2;
        const double a1 = A.kw[c0 + l], a2 = A.kw[TL + c0 + l],
                     a3 = A.kw[2 * TL + c0 + l];
        for (int i = 0; i < A.nfam; i++)
        {
            const int f = A.fam[i];
            const double2 e0 = member(f, n, v0, v1);
            const double2 o = member(f, n + 1, v1, v2);
            const double2 e1 = member(f, n + 2, v2, v3);
            if (A.cs)
            {
                A.cs[i * T1 + t0 + n] = times(A.tc[t0 + n], e0);
                if (n < nmax)
                    A.cs[i * T1 + t0 + n + 1] = times(A.tc[t0 + n + 1], o);
            }
            double2 even = make_double2(fma(a1, e0.x, a2 * e1.x),
                                        fma(a1, e0.y, a2 * e1.y));
            double2 odd = times(a3, o);
            if (f >= 3)
            {
                // the differences G - H, J - N in the other parity's place
                const double2 h0 = member(f - 2, n, v0, v1);
                const double2 h1 = member(f - 2, n + 1, v1, v2);
                const double2 h2 = member(f - 2, n + 2, v2, v3);
                const double2 g = odd;
                odd = make_double2(g.x - fma(a1, h0.x, a2 * h2.x),
                                   g.y - fma(a1, h0.y, a2 * h2.y));
                even = make_double2(even.x - a3 * h1.x, even.y - a3 * h1.y);
            }
            double2 *out = A.cs2 + 2 * (i * TL + c0 + l);
            out[0] = even;
            out[1] = odd;
        }
    }
}

void scale_families(ScaleArgs *A, int mode)
{
    static const int n[] = {1, 2, 4, 3, 5, 5};
    static const int f[][5] = {{0},          {3, 1},          {0, 1, 2, 3},
                               {0, 1, 3},    {0, 1, 2, 3, 4}, {0, 1, 2, 3, 4}};
    A->nfam = n[mode];
    for (int i = 0; i < 5; i++)
        A->fam[i] = f[mode][i];
}

cudaError_t launch_two_tables(long long nmax, const double *sg, double2 *ab,
                              double2 *ag, double *kw, double *sm,
                              cudaStream_t st)
{
    k_two_tables<<<(unsigned)(nmax + 1), TAB_THREADS, 0, st>>>(
        nmax, sg, ab, ag, kw, sm, two_sum(nmax));
    return cudaGetLastError();
}

cudaError_t launch_geometry(const GeometryArgs &G, cudaStream_t st)
{
    const dim3 grid((unsigned)geo_blocks_x(G), (unsigned)geo_blocks_y(G));
    k_geometry<<<grid, GEO_THREADS, 0, st>>>(G);
    return cudaGetLastError();
}

cudaError_t launch_two_scale(const ScaleArgs &A, long long m_lo,
                             long long m_hi, const GeometryArgs *G,
                             cudaStream_t st)
{
    if (m_hi <= m_lo)
        return cudaSuccess;
    const int geo = G ? geo_blocks_x(*G) * geo_blocks_y(*G) : 0;
    k_two_scale<<<(unsigned)(m_hi - m_lo + geo), GEO_THREADS, 0, st>>>(
        A, m_lo, G ? *G : GeometryArgs{}, geo);
    return cudaGetLastError();
}

} // namespace cb
