// Grid synthesis with the two-degree recurrence (two.cuh): the lumped
// coefficients of CHarm's shs_point_kernel
// (src/shs/shs_point_kernel.c:745-2010, driven by shs_point_grd.c:598-1018).
//
// Every quantity is formed from sums F = sum_n F_n P_n of up to five
// coefficient families (k_two_scale), X: C_n, H: n C_n, N: n (n + 1) C_n,
// G: e_n+1 C_n+1, J: (n + 2) e_n+1 C_n+1 (C and S each), by the per-degree
// relations of CHarm's kernels (shs_point_kernel.c:1639-1946) taken out of
// the sums:
//     sum C (n+1) P = H + X,      sum C (n+1)(n+2) P = N + 2 (H + X),
//     sum C dP = (G - t H) / u,   sum C (n+1) dP = (J - t N) / u,
//     sum C ddP = (t / u) sum C dP + (m / u)^2 X - N,
// and near the poles G - t H loses what its two sums have in common.  In the
// two-degree recurrence's pairs, G = E + t O with E = sum e_l s_l, O = sum
// o_l s_l (and H likewise),
//     G - t H = sum (eG_l - oH_l) s_l + u^2 OH + t sum (oG_l - eH_l) s_l,
// upper sign of t north, lower south, so k_two_scale stores the differences
// in the place of eG, oG (and of eJ, oJ with N): what cancels does so in the
// coefficients, degree by degree, as in the one-degree kernel's dP.  Hence a
// degree costs two sums per family and nothing else, where the
// one-degree kernel forms dP, ddP and the degree factors per latitude and
// degree: 10 against 24 FP64 instructions for the second-order gradient, and
// the potential with both gradients (ten quantities) is one pass over the
// same five families instead of three passes.
//
// Bound by the FP64 pipe: per step (two degrees) and latitude pair one DFMA
// for alpha x2 + beta, one for the recurrence and four sums.  The loop alone
// takes 15.3 to 15.7 issue cycles of a sub-partition per step and pair at
// K = 4..6 pairs per lane (12 if no DFMA read three fresh registers), the
// one-degree loop it replaces 19.3 to 20.5 per two degrees.  One warp per
// (order, tile of 32 K pairs), items handed out by an atomic counter in
// order of decreasing cost; K is the autotuner's choice (more pairs amortise
// the staged coefficients, fewer keep more warps resident).  A tile whose
// every latitude is still below the double range runs the recurrence
// without the sums.  Legendre part on B200, before (k_shs_grid) and now:
// GL nmax 1000 0.114 / 0.094 ms, 2190 0.935 / 0.672 ms, 5400 12.6 / 8.6 ms,
// DH2 nmax 719 above the sphere 0.109 / 0.076 ms; ten quantities of eight
// sets at GL nmax 540 (three launches before) 0.806 / 0.368 ms.
#include <cstdint>

#include "common.cuh"
#include "kernels.h"
#include "leg.cuh"
#include "synth.cuh"
#include "two.cuh"

namespace cb
{

namespace
{

// What a kernel forms; families and output quantities of each.
enum
{
    MODE_VALUE = 0,   // the potential and its radial derivatives: X
    MODE_LAT1 = 1,    // first latitudinal derivative: G, H
    MODE_LAT2 = 2,    // second one: X, H, N, G
    MODE_GRAD1 = 3,   // X, H, G
    MODE_GRAD2 = 4,   // X, H, N, G, J
    MODE_TEN = 5      // potential, grad1 and grad2 from the same families
};

constexpr int two_nf(int mode)
{
    return mode == MODE_VALUE ? 1
           : mode == MODE_LAT1 ? 2
           : mode == MODE_LAT2 ? 4
           : mode == MODE_GRAD1 ? 3
                                : 5;
}

// per warp: two stages of (alpha, delta) and the coefficient pairs of every
// family (or, for near_item, beta and the one-degree coefficients of 64
// degrees), two mbarriers
constexpr size_t two_stage(int nf)
{
    return TWO_CHUNK * (1 + 2 * nf) * sizeof(double2);
}
constexpr size_t near_stage(int nf)
{
    return LEG_CHUNK * (1 + nf) * sizeof(double2);
}
constexpr size_t two_warp_smem(int nf)
{
    return 2 * near_stage(nf) + 2 * sizeof(uint64_t);
}
static_assert(near_stage(5) >= two_stage(5), "the larger stage sets the size");

// resident blocks per SM at which each tile width stays free of spills
constexpr int two_min_blocks(int nf, int K)
{
    if (nf == 1)
        return K >= 5 ? 3 : 4;
    return nf * K >= 8 ? 2 : (nf * K >= 5 ? 3 : 4);
}

// The common end of an item: the lumped coefficients of pair p from the sums
// over the two parities of n - m, acc[family][C, S][even, odd]: of the
// two-degree recurrence (`two`: odd sums without the factor sin(lat), G and J
// as differences) or of near_item.
template <int MODE>
__device__ __forceinline__ void two_store(
    const ShsTwoArgs &A, double2 *outp, long long m, const double (&mur)[3],
    int p, const double (&acc)[two_nf(MODE)][2][2], bool two)
{
    constexpr int NF = two_nf(MODE);
    const double md = (double)m;
    const double cpack = A.fft_pack ? (m == 0 ? 1.0 : 0.5) : 1.0;
    const double sgnb = A.fft_pack ? -1.0 : 1.0;
    const double t = A.t[p];
    const double ur = MODE == MODE_VALUE && !A.dlon ? 1.0 : 1.0 / A.u[p];
    const double u2 = ur * ur;
#pragma unroll
    for (int h = 0; h < 2; h++)
    {
        const int row = h == 0 ? A.row_n[p] : A.row_s[p];
        if (row < 0 || row >= A.nlat)
            continue;
        const double th = h == 0 ? t : -t, tuh = th * ur;
        double F[NF][2];
#pragma unroll
        for (int f = 0; f < NF; f++)
#pragma unroll
            for (int i = 0; i < 2; i++)
            {
                const double o = two ? __dmul_rn(t, acc[f][i][1])
                                     : acc[f][i][1];
                F[f][i] = h == 0 ? __dadd_rn(acc[f][i][0], o)
                                 : __dsub_rn(acc[f][i][0], o);
            }
        auto put = [&](int q, double mu, double a, double b) {
            outp[((size_t)q * A.nlat + row) * (size_t)A.ldf + m] =
                make_double2(cpack * mu * a, sgnb * (cpack * mu * b));
        };
        // explicit operations: the same bits whichever kernel forms them.
        // d1(g, h, i): (G - t H) / u of the families g and h
        auto d1 = [&](int g, int hf, int i) {
            const double x =
                two ? __fma_rn(__dmul_rn(A.u[p], A.u[p]), acc[hf][i][1],
                               F[g][i])
                    : __fma_rn(-th, F[hf][i], F[g][i]);
            return __dmul_rn(ur, x);
        };
        auto d2 = [&](double x, double n, double d) {
            const double w = __dmul_rn(__dmul_rn(md, md), u2);
            return __dsub_rn(__fma_rn(w, x, __dmul_rn(tuh, d)), n);
        };
        if constexpr (MODE <= MODE_LAT2)
        {
            double a[1], b[1];
            if constexpr (MODE == MODE_VALUE)
            {
                a[0] = F[0][0];
                b[0] = F[0][1];
            }
            else if constexpr (MODE == MODE_LAT1)
            {
                a[0] = d1(0, 1, 0);
                b[0] = d1(0, 1, 1);
            }
            else
            {
                a[0] = d2(F[0][0], F[2][0], d1(3, 1, 0));
                b[0] = d2(F[0][1], F[2][1], d1(3, 1, 1));
            }
            if (A.dr == 1)
                lumped_post<0, 1, 1>(a, b, md, ur, u2, tuh, A.dlon);
            else
                lumped_post<0, 0, 1>(a, b, md, ur, u2, tuh, A.dlon);
            put(0, mur[0], a[0], b[0]);
        }
        if constexpr (MODE == MODE_TEN)
            put(0, mur[0], F[0][0], F[0][1]);
        if constexpr (MODE == MODE_GRAD1 || MODE == MODE_TEN)
        {
            constexpr int G = MODE == MODE_TEN ? 3 : 2;
            constexpr int q0 = MODE == MODE_TEN ? 1 : 0;
            double a[3] = {F[0][0], __dadd_rn(F[1][0], F[0][0]),
                           d1(G, 1, 0)};
            double b[3] = {F[0][1], __dadd_rn(F[1][1], F[0][1]),
                           d1(G, 1, 1)};
            lumped_post<1, 0, 3>(a, b, md, ur, u2, tuh, A.dlon);
#pragma unroll
            for (int q = 0; q < 3; q++)
                put(q0 + q, mur[MODE == MODE_TEN ? 1 : 0], a[q], b[q]);
        }
        if constexpr (MODE == MODE_GRAD2 || MODE == MODE_TEN)
        {
            constexpr int q0 = MODE == MODE_TEN ? 4 : 0;
            double v[2][6];
#pragma unroll
            for (int i = 0; i < 2; i++)
            {
                const double x = F[0][i], n = F[2][i];
                const double p1 = __dadd_rn(F[1][i], x);
                const double d = d1(3, 1, i);
                v[i][0] = x;
                v[i][1] = p1;
                v[i][2] = d;
                v[i][3] = __fma_rn(2.0, p1, n);
                v[i][4] = d1(4, 2, i);
                v[i][5] = d2(x, n, d);
            }
            lumped_post<2, 0, 6>(v[0], v[1], md, ur, u2, tuh, A.dlon);
#pragma unroll
            for (int q = 0; q < 6; q++)
                put(q0 + q, mur[MODE == MODE_TEN ? 2 : 0], v[0][q], v[1][q]);
        }
    }
}

// One order of a tile of 32 NEAR_K pairs next to the equator: the one-degree
// recurrence of leg.cuh, staged through the same ring.  These items are the
// longest chains of the launch (one dependent DFMA per degree instead of one
// per two) and a few per cent of its work; each order's come first.
constexpr int NEAR_K = SHS_NEAR_PAIRS / 32;

template <int MODE>
__device__ __noinline__ bool near_item(const ShsTwoArgs &A, long long m,
                                       int tile, long long Nset,
                                       const double2 *cs1, double2 *outp,
                                       const double (&mur)[3],
                                       double polar_thr, unsigned char *smem,
                                       uint64_t *bar, unsigned &phases)
{
    constexpr int NF = two_nf(MODE);
    const unsigned lane = threadIdx.x & 31u;
    double t[NEAR_K], x[NEAR_K], y[NEAR_K], acc[NEAR_K][NF][2][2];
    int E[NEAR_K];
    bool skip = polar_thr >= 0.0, any_scaled = false;
#pragma unroll
    for (int k = 0; k < NEAR_K; k++)
    {
        const int i = tile * (32 * NEAR_K) + k * 32 + (int)lane;
        const bool valid = i < A.nnear;
        const int p = A.near0 + i;
        t[k] = valid ? A.t[p] : 0.0;
        x[k] = y[k] = 0.0;
        E[k] = 0;
        if (valid)
        {
            two_seed(A.pw, A.pw_ld, p, m, A.sg[2 * m], y[k], E[k]);
            if (!((double)m - (double)Nset * A.u[p] > polar_thr))
                skip = false;
        }
        any_scaled |= E[k] != 0;
#pragma unroll
        for (int f = 0; f < NF; f++)
            acc[k][f][0][0] = acc[k][f][0][1] = acc[k][f][1][0] =
                acc[k][f][1][1] = 0.0;
    }
    skip = __all_sync(0xffffffffu, skip);
    any_scaled = __any_sync(0xffffffffu, any_scaled);
    if (!skip)
    {
        const long long c0 = tri_col0(A.nmax, m);
        const long long T1 = tri_size(A.nmax);
        const int ncol = (int)(Nset - m + 1);
        const int nchunks = (ncol + LEG_CHUNK - 1) / LEG_CHUNK;
        auto stage = [&](int s) {
            return reinterpret_cast<double2 *>(smem + s * near_stage(NF));
        };
        auto issue = [&](int j, int s) {
            if (lane == 0)
            {
                const unsigned bytes =
                    (unsigned)(min(ncol - j * LEG_CHUNK, LEG_CHUNK) *
                               sizeof(double2));
                mbar_arrive_expect_tx(&bar[s], (1 + NF) * bytes);
                bulk_g2s(stage(s), A.tb + c0 + j * LEG_CHUNK, bytes, &bar[s]);
#pragma unroll
                for (int f = 0; f < NF; f++)
                    bulk_g2s(stage(s) + (1 + f) * LEG_CHUNK,
                             cs1 + f * T1 + c0 + j * LEG_CHUNK, bytes,
                             &bar[s]);
            }
        };
        __syncwarp();
        fence_proxy_async_smem();
        issue(0, 0);
        if (nchunks > 1)
            issue(1, 1);
        for (int j = 0; j < nchunks; j++)
        {
            const int s = j & 1;
            const int cnt = min(ncol - j * LEG_CHUNK, LEG_CHUNK);
            if (!mbar_wait_bounded(&bar[s], (phases >> s) & 1u, A.status))
                return false;
            phases ^= 1u << s;
            double2 *stb = stage(s);
            const double2 *scs = stb + LEG_CHUNK;
            if (j > 0)
            {
                const double mul = A.tmul[(size_t)m * A.ldmul + j];
#pragma unroll
                for (int k = 0; k < NEAR_K; k++)
                {
                    x[k] *= mul;
                    y[k] *= mul;
                }
            }
            else
            {
                if (lane == 0)
                    stb[0].x = -1.0;   // the first step yields the seed (in y)
                __syncwarp();
            }
            auto step = [&](int i, int par) {
                const double beta = stb[i].x;
#pragma unroll
                for (int k = 0; k < NEAR_K; k++)
                {
                    const double v = fma(t[k], x[k], -(beta * y[k]));
                    y[k] = x[k];
                    x[k] = v;
                }
#pragma unroll
                for (int f = 0; f < NF; f++)
                {
                    const double2 c = scs[f * LEG_CHUNK + i];
#pragma unroll
                    for (int k = 0; k < NEAR_K; k++)
                    {
                        acc[k][f][0][par] = fma(x[k], c.x, acc[k][f][0][par]);
                        acc[k][f][1][par] = fma(x[k], c.y, acc[k][f][1][par]);
                    }
                }
            };
            int i = 0;
#pragma unroll(NF == 1 ? 8 : 2)
            for (; i + 1 < cnt; i += 2)
            {
                step(i, 0);
                step(i + 1, 1);
            }
            if (i < cnt)
                step(i, 0);
            if (any_scaled)
            {
                bool still = false;
#pragma unroll
                for (int k = 0; k < NEAR_K; k++)
                {
                    if (leg_fixup(x[k], y[k], E[k]))
                    {
#pragma unroll
                        for (int f = 0; f < NF; f++)
                            acc[k][f][0][0] = acc[k][f][0][1] =
                                acc[k][f][1][0] = acc[k][f][1][1] = 0.0;
                    }
                    still |= E[k] != 0;
                }
                any_scaled = __any_sync(0xffffffffu, still);
            }
            __syncwarp();
            if (j + 2 < nchunks)
            {
                fence_proxy_async_smem();
                issue(j + 2, s);
            }
        }
    }
#pragma unroll
    for (int k = 0; k < NEAR_K; k++)
    {
        const int i = tile * (32 * NEAR_K) + k * 32 + (int)lane;
        if (i >= A.nnear)
            continue;
        if (E[k] != 0 || skip)
        {
#pragma unroll
            for (int f = 0; f < NF; f++)
                acc[k][f][0][0] = acc[k][f][0][1] = acc[k][f][1][0] =
                    acc[k][f][1][1] = 0.0;
        }
        two_store<MODE>(A, outp, m, mur, A.near0 + i, acc[k], false);
    }
    __syncwarp();
    return true;
}

} // namespace

template <int MODE, int K>
__global__ void __launch_bounds__(128, two_min_blocks(two_nf(MODE), K))
    k_shs_two(const __grid_constant__ ShsTwoArgs A)
{
    constexpr int NF = two_nf(MODE);
    extern __shared__ __align__(128) unsigned char smem_raw[];
    const unsigned lane = threadIdx.x & 31u;
    const unsigned warp = threadIdx.x >> 5;
    unsigned char *wbase = smem_raw + (size_t)warp * two_warp_smem(NF);
    uint64_t *bar = reinterpret_cast<uint64_t *>(wbase + 2 * near_stage(NF));
    auto stg = [&](int s) {
        return reinterpret_cast<double2 *>(wbase + (size_t)s * two_stage(NF));
    };
    if (lane == 0)
    {
        mbar_init(&bar[0], 1);
        mbar_init(&bar[1], 1);
        fence_mbar_init();
    }
    __syncwarp();
    unsigned phases = 0u;
    const long long N = A.nmax;
    const int np = A.npairs;

    for (;;)
    {
        unsigned long long item = 0;
        if (lane == 0)
            item = atomicAdd(A.counter, 1ull);
        item = __shfl_sync(0xffffffffu, item, 0);
        if (item >= (unsigned long long)A.nitems)
            break;
        // batched sets: items of set j start at sets[j].item0
        long long Nset = N;
        const double2 *csp = A.cs, *cs1 = A.cs1;
        double2 *outp = A.out;
        double mur[3] = {A.mur, 0.0, 0.0}, polar_thr = A.polar_thr;
        unsigned long long local = item;
        if (A.nsets > 0)
        {
            int lo = 0, hi = A.nsets - 1;
            while (lo < hi)
            {
                const int mid = (lo + hi + 1) >> 1;
                if ((unsigned long long)A.sets[mid].item0 <= item)
                    lo = mid;
                else
                    hi = mid - 1;
            }
            const BatchSet &bs = A.sets[lo];
            Nset = bs.nmax;
            csp = bs.cs;
            cs1 = bs.cs1;
            outp = bs.out;
            mur[0] = bs.mur;
            mur[1] = bs.mur1;
            mur[2] = bs.mur2;
            polar_thr = bs.polar_thr;
            local = item - (unsigned long long)bs.item0;
        }
        const unsigned per = (unsigned)(A.ntiles + A.near_tiles);
        const long long m = A.m0 + (long long)((unsigned)local / per);
        const int sub = (int)((unsigned)local % per);
        if (sub < A.near_tiles)
        {
            if (!near_item<MODE>(A, m, sub, Nset, cs1, outp, mur, polar_thr,
                                 wbase, &bar[0], phases))
                break;
            continue;
        }
        const int tile = A.tile0 + sub - A.near_tiles;
        const double sigma = A.sm[m];

        double z[K], x[K], y[K];
        int E[K];
        bool polar_skip = polar_thr >= 0.0;
#pragma unroll
        for (int k = 0; k < K; k++)
        {
            const int p = tile * (32 * K) + k * 32 + (int)lane;
            const bool valid = p < np;
            const double u = valid ? A.u[p] : 1.0;
            z[k] = valid ? A.z[p] : 0.0;
            y[k] = 0.0;
            x[k] = 0.0;
            E[k] = 0;
            if (valid)
            {
                two_seed(A.pw, A.pw_ld, p, m, sigma, x[k], E[k]);
                if (!((double)m - (double)Nset * u > polar_thr))
                    polar_skip = false;
            }
        }
        polar_skip = __all_sync(0xffffffffu, polar_skip);

        double acc[K][NF][2][2];   // [family][C, S][even, odd]
        auto zero = [&](int k) {
#pragma unroll
            for (int f = 0; f < NF; f++)
                acc[k][f][0][0] = acc[k][f][0][1] = acc[k][f][1][0] =
                    acc[k][f][1][1] = 0.0;
        };
#pragma unroll
        for (int k = 0; k < K; k++)
            zero(k);

        if (!polar_skip)
        {
            const long long c0 = two_col0(N, m);
            const long long T2 = 2 * two_sum(N);
            const int nl = (int)two_len(Nset, m);
            const int nchunks = (nl + TWO_CHUNK - 1) / TWO_CHUNK;
            // pairs below A.polar (a multiple of 32) take the polar form;
            // tiles on the border read (alpha, beta) and add alpha for them
            const int g0 = tile * (32 * K);
            const bool mixed = g0 < A.polar && g0 + 32 * K > A.polar;
            const double2 *tab = g0 + 32 * K <= A.polar ? A.ag : A.ab;
            auto issue = [&](int j, int s) {
                if (lane == 0)
                {
                    const long long off = c0 + (long long)j * TWO_CHUNK;
                    const int cnt = min(nl - j * TWO_CHUNK, TWO_CHUNK);
                    const unsigned bytes = (unsigned)(cnt * sizeof(double2));
                    mbar_arrive_expect_tx(&bar[s], (1 + 2 * NF) * bytes);
                    bulk_g2s(stg(s), tab + off, bytes, &bar[s]);
#pragma unroll
                    for (int f = 0; f < NF; f++)
                        bulk_g2s(stg(s) + (1 + 2 * f) * TWO_CHUNK,
                                 csp + f * T2 + 2 * off, 2 * bytes, &bar[s]);
                }
            };
            // the warp's earlier accesses to the stages before these copies
            __syncwarp();
            fence_proxy_async_smem();
            issue(0, 0);
            if (nchunks > 1)
                issue(1, 1);
            bool any_scaled = false, any_live = false;
#pragma unroll
            for (int k = 0; k < K; k++)
            {
                any_scaled |= E[k] != 0;
                any_live |= E[k] == 0 && x[k] != 0.0;
            }
            any_scaled = __any_sync(0xffffffffu, any_scaled);
            any_live = __any_sync(0xffffffffu, any_live);

            bool ok = true;
            for (int j = 0; j < nchunks; j++)
            {
                const int s = j & 1;
                if (!mbar_wait_bounded(&bar[s], (phases >> s) & 1u, A.status))
                {
                    ok = false;
                    break;
                }
                phases ^= 1u << s;
                const int cnt = min(nl - j * TWO_CHUNK, TWO_CHUNK);
                const double2 *sab = stg(s);
                const double2 *scs = stg(s) + TWO_CHUNK;
                auto sums = [&](int i) {
#pragma unroll
                    for (int f = 0; f < NF; f++)
                    {
                        const double2 ce = scs[2 * f * TWO_CHUNK + 2 * i];
                        const double2 co = scs[2 * f * TWO_CHUNK + 2 * i + 1];
#pragma unroll
                        for (int k = 0; k < K; k++)
                        {
                            double (&v)[2][2] = acc[k][f];
                            v[0][0] = fma(x[k], ce.x, v[0][0]);
                            v[1][0] = fma(x[k], ce.y, v[1][0]);
                            v[0][1] = fma(x[k], co.x, v[0][1]);
                            v[1][1] = fma(x[k], co.y, v[1][1]);
                        }
                    }
                };
                auto advance = [&](int i) {
                    const double2 ab = sab[i];
#pragma unroll
                    for (int k = 0; k < K; k++)
                    {
                        const double f = fma(ab.x, z[k], ab.y);
                        const double xn = fma(f, x[k], -y[k]);
                        y[k] = x[k];
                        x[k] = xn;
                    }
                };
                auto advance_mixed = [&](int i) {
                    const double2 ab = sab[i];
                    const double g = ab.x + ab.y;
#pragma unroll
                    for (int k = 0; k < K; k++)
                    {
                        const double f = fma(
                            ab.x, z[k], g0 + 32 * k < A.polar ? g : ab.y);
                        const double xn = fma(f, x[k], -y[k]);
                        y[k] = x[k];
                        x[k] = xn;
                    }
                };
                if (any_live && !mixed && cnt == TWO_CHUNK)
                {
#pragma unroll(NF <= 2 ? 4 : 2)
                    for (int i = 0; i < TWO_CHUNK; i++)
                    {
                        sums(i);
                        advance(i);
                    }
                }
                else if (any_live && !mixed)
                {
#pragma unroll 2
                    for (int i = 0; i < cnt; i++)
                    {
                        sums(i);
                        advance(i);
                    }
                }
                else if (any_live)
                {
#pragma unroll 2
                    for (int i = 0; i < cnt; i++)
                    {
                        sums(i);
                        advance_mixed(i);
                    }
                }
                else if (!mixed)
                {
#pragma unroll 4
                    for (int i = 0; i < cnt; i++)
                        advance(i);
                }
                else
                {
#pragma unroll 2
                    for (int i = 0; i < cnt; i++)
                        advance_mixed(i);
                }
                if (any_scaled)
                {
                    bool still = false, live = false;
#pragma unroll
                    for (int k = 0; k < K; k++)
                    {
                        if (two_fixup(x[k], y[k], E[k]))
                            zero(k);
                        still |= E[k] != 0;
                        live |= E[k] == 0 && x[k] != 0.0;
                    }
                    any_scaled = __any_sync(0xffffffffu, still);
                    any_live |= __any_sync(0xffffffffu, live);
                }
                __syncwarp();
                if (j + 2 < nchunks)
                {
                    fence_proxy_async_smem();
                    issue(j + 2, s);
                }
            }
            if (!ok)
                break;
            // latitudes that never left the scaled range contribute nothing
#pragma unroll
            for (int k = 0; k < K; k++)
                if (E[k] != 0)
                    zero(k);
        }

#pragma unroll
        for (int k = 0; k < K; k++)
        {
            const int p = tile * (32 * K) + k * 32 + (int)lane;
            if (p >= np)
                continue;
            two_store<MODE>(A, outp, m, mur, p, acc[k], true);
        }
    }
}

template <int MODE, int K>
static cudaError_t launch_one(const ShsTwoArgs &A, int grid, cudaStream_t st)
{
    const int warps = 4;
    constexpr size_t smem = warps * two_warp_smem(two_nf(MODE));
    if constexpr (smem > 48 * 1024)
    {
        static const cudaError_t attr = cudaFuncSetAttribute(
            (const void *)k_shs_two<MODE, K>,
            cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (attr != cudaSuccess)
            return attr;
    }
    k_shs_two<MODE, K><<<grid, warps * 32, smem, st>>>(A);
    return cudaGetLastError();
}

template <int MODE>
static cudaError_t launch_mode(const ShsTwoArgs &A, int K, int grid,
                               cudaStream_t st)
{
    if constexpr (MODE == MODE_VALUE)
    {
        switch (K)
        {
        case 6: return launch_one<MODE, 6>(A, grid, st);
        case 5: return launch_one<MODE, 5>(A, grid, st);
        case 4: return launch_one<MODE, 4>(A, grid, st);
        case 3: return launch_one<MODE, 3>(A, grid, st);
        default: break;
        }
    }
    if (K > 2)
        return cudaErrorInvalidValue;
    return K == 2 ? launch_one<MODE, 2>(A, grid, st)
                  : launch_one<MODE, 1>(A, grid, st);
}

cudaError_t launch_shs_two(const ShsTwoArgs &A, int K, int grid,
                           cudaStream_t st)
{
    switch (A.mode)
    {
    case MODE_VALUE: return launch_mode<MODE_VALUE>(A, K, grid, st);
    case MODE_LAT1: return launch_mode<MODE_LAT1>(A, K, grid, st);
    case MODE_LAT2: return launch_mode<MODE_LAT2>(A, K, grid, st);
    case MODE_GRAD1: return launch_mode<MODE_GRAD1>(A, K, grid, st);
    case MODE_GRAD2: return launch_mode<MODE_GRAD2>(A, K, grid, st);
    case MODE_TEN: return launch_mode<MODE_TEN>(A, K, grid, st);
    default: return cudaErrorInvalidValue;
    }
}

} // namespace cb
