// Grid synthesis with the two-degree recurrence (two.cuh): the lumped
// coefficients of CHarm's shs_point_kernel
// (src/shs/shs_point_kernel.c:745-2010, driven by shs_point_grd.c:598-1018)
// for the potential and the radial derivatives.
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
// DH2 nmax 719 above the sphere 0.109 / 0.076 ms.
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

// per warp: two stages of (alpha, delta) and the coefficient pairs, two
// mbarriers
constexpr size_t TWO_STAGE = TWO_CHUNK * 3 * sizeof(double2);
constexpr size_t NEAR_STAGE = 2 * LEG_CHUNK * sizeof(double2);
constexpr size_t TWO_WARP_SMEM = 2 * NEAR_STAGE + 2 * sizeof(uint64_t);
static_assert(NEAR_STAGE >= TWO_STAGE, "the larger stage sets the size");

// resident blocks per SM at which each tile width stays free of spills
constexpr int two_min_blocks(int K) { return K >= 7 ? 2 : (K >= 5 ? 3 : 4); }

// The common end of an item: the lumped coefficients of pair p from the sums
// over the two parities of n - m (odd: times sin(lat) already).
__device__ __forceinline__ void two_store(const ShsTwoArgs &A, double2 *outp,
                                          long long m, double mur, int p,
                                          double ec, double es, double oc,
                                          double os)
{
    const double md = (double)m;
    const double cpack = A.fft_pack ? (m == 0 ? 1.0 : 0.5) : 1.0;
    const double sgnb = A.fft_pack ? -1.0 : 1.0;
    const double ur = A.dlon ? 1.0 / A.u[p] : 1.0;
#pragma unroll
    for (int h = 0; h < 2; h++)
    {
        const int row = h == 0 ? A.row_n[p] : A.row_s[p];
        if (row < 0 || row >= A.nlat)
            continue;
        double a[1] = {h == 0 ? ec + oc : ec - oc};
        double b[1] = {h == 0 ? es + os : es - os};
        if (A.dr == 1)
            lumped_post<0, 1, 1>(a, b, md, ur, ur * ur, 0.0, A.dlon);
        else
            lumped_post<0, 0, 1>(a, b, md, ur, ur * ur, 0.0, A.dlon);
        outp[(size_t)row * (size_t)A.ldf + m] =
            make_double2(cpack * mur * a[0], sgnb * (cpack * mur * b[0]));
    }
}

// One order of a tile of 32 NEAR_K pairs next to the equator: the one-degree
// recurrence of leg.cuh, staged through the same ring.  These items are the
// longest chains of the launch (one dependent DFMA per degree instead of one
// per two) and a few per cent of its work; each order's come first.
constexpr int NEAR_K = SHS_NEAR_PAIRS / 32;

__device__ __noinline__ bool near_item(const ShsTwoArgs &A, long long m,
                                       int tile, long long Nset,
                                       const double2 *cs1, double2 *outp,
                                       double mur, double polar_thr,
                                       unsigned char *smem, uint64_t *bar,
                                       unsigned &phases)
{
    const unsigned lane = threadIdx.x & 31u;
    double t[NEAR_K], x[NEAR_K], y[NEAR_K], acc[NEAR_K][2][2];
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
        acc[k][0][0] = acc[k][0][1] = acc[k][1][0] = acc[k][1][1] = 0.0;
    }
    skip = __all_sync(0xffffffffu, skip);
    any_scaled = __any_sync(0xffffffffu, any_scaled);
    if (!skip)
    {
        const long long c0 = tri_col0(A.nmax, m);
        const int ncol = (int)(Nset - m + 1);
        const int nchunks = (ncol + LEG_CHUNK - 1) / LEG_CHUNK;
        auto stage = [&](int s) {
            return reinterpret_cast<double2 *>(smem + s * NEAR_STAGE);
        };
        auto issue = [&](int j, int s) {
            if (lane == 0)
            {
                const unsigned bytes =
                    (unsigned)(min(ncol - j * LEG_CHUNK, LEG_CHUNK) *
                               sizeof(double2));
                mbar_arrive_expect_tx(&bar[s], 2 * bytes);
                bulk_g2s(stage(s), A.tb + c0 + j * LEG_CHUNK, bytes, &bar[s]);
                bulk_g2s(stage(s) + LEG_CHUNK, cs1 + c0 + j * LEG_CHUNK,
                         bytes, &bar[s]);
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
                const double2 c = scs[i];
#pragma unroll
                for (int k = 0; k < NEAR_K; k++)
                {
                    const double v = fma(t[k], x[k], -(beta * y[k]));
                    y[k] = x[k];
                    x[k] = v;
                    acc[k][0][par] = fma(v, c.x, acc[k][0][par]);
                    acc[k][1][par] = fma(v, c.y, acc[k][1][par]);
                }
            };
            int i = 0;
#pragma unroll 8
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
                        acc[k][0][0] = acc[k][0][1] = acc[k][1][0] =
                            acc[k][1][1] = 0.0;
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
        const double live = E[k] == 0 && !skip ? 1.0 : 0.0;
        two_store(A, outp, m, mur, A.near0 + i, live * acc[k][0][0],
                  live * acc[k][1][0], live * acc[k][0][1],
                  live * acc[k][1][1]);
    }
    __syncwarp();
    return true;
}

} // namespace

template <int K>
__global__ void __launch_bounds__(128, two_min_blocks(K))
    k_shs_two(const __grid_constant__ ShsTwoArgs A)
{
    extern __shared__ __align__(128) unsigned char smem_raw[];
    const unsigned lane = threadIdx.x & 31u;
    const unsigned warp = threadIdx.x >> 5;
    unsigned char *wbase = smem_raw + (size_t)warp * TWO_WARP_SMEM;
    uint64_t *bar = reinterpret_cast<uint64_t *>(wbase + 2 * NEAR_STAGE);
    auto stg = [&](int s) {
        return reinterpret_cast<double2 *>(wbase + (size_t)s * TWO_STAGE);
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
        double mur = A.mur, polar_thr = A.polar_thr;
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
            mur = bs.mur;
            polar_thr = bs.polar_thr;
            local = item - (unsigned long long)bs.item0;
        }
        const unsigned per = (unsigned)(A.ntiles + A.near_tiles);
        const long long m = A.m0 + (long long)((unsigned)local / per);
        const int sub = (int)((unsigned)local % per);
        if (sub < A.near_tiles)
        {
            if (!near_item(A, m, sub, Nset, cs1, outp, mur, polar_thr, wbase,
                           &bar[0], phases))
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

        double ec[K], es[K], oc[K], os[K];
#pragma unroll
        for (int k = 0; k < K; k++)
            ec[k] = es[k] = oc[k] = os[k] = 0.0;

        if (!polar_skip)
        {
            const long long c0 = two_col0(N, m);
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
                    mbar_arrive_expect_tx(&bar[s], 3 * bytes);
                    bulk_g2s(stg(s), tab + off, bytes, &bar[s]);
                    bulk_g2s(stg(s) + TWO_CHUNK, csp + 2 * off, 2 * bytes,
                             &bar[s]);
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
                    const double2 ce = scs[2 * i], co = scs[2 * i + 1];
#pragma unroll
                    for (int k = 0; k < K; k++)
                    {
                        ec[k] = fma(x[k], ce.x, ec[k]);
                        es[k] = fma(x[k], ce.y, es[k]);
                        oc[k] = fma(x[k], co.x, oc[k]);
                        os[k] = fma(x[k], co.y, os[k]);
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
#pragma unroll 4
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
                            ec[k] = es[k] = oc[k] = os[k] = 0.0;
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
                    ec[k] = es[k] = oc[k] = os[k] = 0.0;
        }

#pragma unroll
        for (int k = 0; k < K; k++)
        {
            const int p = tile * (32 * K) + k * 32 + (int)lane;
            if (p >= np)
                continue;
            const double t = A.t[p];
            two_store(A, outp, m, mur, p, ec[k], es[k], t * oc[k], t * os[k]);
        }
    }
}

template <int K>
static cudaError_t launch_one(const ShsTwoArgs &A, int grid, cudaStream_t st)
{
    const int warps = 4;
    const size_t smem = (size_t)warps * TWO_WARP_SMEM;
    k_shs_two<K><<<grid, warps * 32, smem, st>>>(A);
    return cudaGetLastError();
}

cudaError_t launch_shs_two(const ShsTwoArgs &A, int K, int grid,
                           cudaStream_t st)
{
    switch (K)
    {
    case 8: return launch_one<8>(A, grid, st);
    case 7: return launch_one<7>(A, grid, st);
    case 6: return launch_one<6>(A, grid, st);
    case 5: return launch_one<5>(A, grid, st);
    case 4: return launch_one<4>(A, grid, st);
    case 3: return launch_one<3>(A, grid, st);
    case 2: return launch_one<2>(A, grid, st);
    default: return launch_one<1>(A, grid, st);
    }
}

} // namespace cb
