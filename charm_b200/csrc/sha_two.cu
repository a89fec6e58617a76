// Grid analysis with the two-degree recurrence (two.cuh): the per-order
// Legendre contraction of CHarm's sha_point (src/sha/sha_point.c:713-980)
// after the r2c transform of the grid rows.
//
// Work item = (order m, group g of latitude tiles); one warp per item, K
// latitude pairs per lane.  Per step (two degrees) a lane forms the partial
// sums over its pairs of s_l times the even and odd amplitudes (C and S
// each; the odd ones carry sin(lat)); sixteen steps fill a padded 32 x 33
// array in shared memory whose rows the lanes then add up, and the warp adds
// the totals to the group's partial column.  Per step and pair 6 FP64
// instructions (8 in the one-degree kernel), and per step, whatever K, 4
// additions and 2 KB through the shared-memory port, 64 of about 80 issue
// cycles at K = 4: the port and the FP64 pipe share the limit.  The pairs
// next to the equator form one more group per order, by the one-degree
// recurrence.  k_two_reduce adds the groups in a fixed order, applies k_l and
// combines neighbouring q's into the even degrees: results are
// deterministic.  Legendre part on B200, before (k_sha_grid) and now: GL
// nmax 1000 0.175 / 0.125 ms, 2190 1.125 / 0.886 ms, 5400 15.6 / 11.2 ms,
// DH2 nmax 719 0.144 / 0.097 ms.
#include <cstdint>
#include <type_traits>

#include "common.cuh"
#include "kernels.h"
#include "leg.cuh"
#include "two.cuh"

namespace cb
{

namespace
{

// Partial sums of RED_ROWS (step, parity) or degrees per lane: rows of 32
// lanes, RED_LD apart, so that the row-wise stores and the read-back (lane
// l adds row l) are free of bank conflicts.  (Sixteen rows, for four blocks
// per SM instead of three, was 3 to 7% slower: the shared-memory port is the
// limit, 82% busy at K = 4.)
constexpr int RED_ROWS = 32, RED_LD = 33;
// per warp: two stages, two mbarriers, the partial sums
constexpr size_t SHA_STAGE = LEG_CHUNK * sizeof(double2);
static_assert(SHA_STAGE >= TWO_CHUNK * sizeof(double2), "stage size");
constexpr size_t SHA_WARP_SMEM =
    2 * SHA_STAGE + 16 + RED_ROWS * RED_LD * sizeof(double2);

struct PairAmp
{
    double ae, ao, be, bo;
};

// amplitudes of pair p: even and odd parts of the weighted spectra of its
// two rows (sha_point.c:740-747)
__device__ __forceinline__ PairAmp load_amp(const ShaTwoArgs &A, int p,
                                            long long m)
{
    PairAmp r;
    const int rn = A.row_n[p], rs = A.row_s[p];
    const double2 Fn = A.F[(size_t)rn * A.ldF + m];
    const double a = A.cw_n[p] * Fn.x, b = -A.cw_n[p] * Fn.y;
    double a2 = 0.0, b2 = 0.0;
    if (rs >= 0)
    {
        const double2 Fs = A.F[(size_t)rs * A.ldF + m];
        a2 = A.cw_s[p] * Fs.x;
        b2 = -A.cw_s[p] * Fs.y;
    }
    r.ae = a + a2;
    r.ao = a - a2;
    r.be = b + b2;
    r.bo = b - b2;
    return r;
}

// Lane l's total of row l (fixed order).
__device__ __forceinline__ double2 row_total(const double2 *red, unsigned lane)
{
    const double2 *row = red + lane * RED_LD;
    double c0 = 0.0, s0 = 0.0, c1 = 0.0, s1 = 0.0;
#pragma unroll
    for (int q = 0; q < 32; q += 2)
    {
        const double2 a = row[q], b = row[q + 1];
        c0 += a.x;
        s0 += a.y;
        c1 += b.x;
        s1 += b.y;
    }
    return make_double2(c0 + c1, s0 + s1);
}

// The order's column of the equatorial pairs, one pair per lane and 32 pairs
// after another, by the one-degree recurrence (as k_sha_grid).
__device__ __noinline__ bool near_column(const ShaTwoArgs &A, long long m,
                                         unsigned char *wbase, uint64_t *bar,
                                         double2 *red, unsigned &phases)
{
    const unsigned lane = threadIdx.x & 31u;
    const long long N = A.nmax;
    const long long c0 = tri_col0(N, m);
    const int ncol = (int)(N - m + 1);
    const int nchunks = (ncol + LEG_CHUNK - 1) / LEG_CHUNK;
    double2 *col = A.part1 + c0;
    bool stored = false;
    auto stg = [&](int s) {
        return reinterpret_cast<double2 *>(wbase + (size_t)s * SHA_STAGE);
    };
    for (int i0 = 0; i0 < A.nnear; i0 += 32)
    {
        const bool valid = i0 + (int)lane < A.nnear;
        const int p = A.near0 + i0 + (int)lane;
        double t = 0.0, x = 0.0, y = 0.0;
        int E = 0;
        PairAmp pa{0.0, 0.0, 0.0, 0.0};
        bool skip = A.polar_thr >= 0.0;
        if (valid)
        {
            t = A.t[p];
            two_seed(A.pw, A.pw_ld, p, m, A.sg[2 * m], y, E);
            if (!((double)m - (double)N * A.u[p] > A.polar_thr))
                skip = false;
            if (E == 0)
                pa = load_amp(A, p, m);
        }
        if (__all_sync(0xffffffffu, skip))
            continue;
        bool any_scaled = __any_sync(0xffffffffu, E != 0);
        auto issue = [&](int j, int s) {
            if (lane == 0)
            {
                const unsigned bytes =
                    (unsigned)(min(ncol - j * LEG_CHUNK, LEG_CHUNK) *
                               sizeof(double2));
                mbar_arrive_expect_tx(&bar[s], bytes);
                bulk_g2s(stg(s), A.tb + c0 + j * LEG_CHUNK, bytes, &bar[s]);
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
            if (!mbar_wait_bounded(&bar[s], (phases >> s) & 1u, A.status))
                return false;
            phases ^= 1u << s;
            if (j > 0)
            {
                const double mul = A.tmul[(size_t)m * A.ldmul + j];
                x *= mul;
                y *= mul;
            }
            const int cnt = min(ncol - j * LEG_CHUNK, LEG_CHUNK);
            double2 *stb = stg(s);
            // degrees beyond nmax read beta = 0 and contribute nothing that
            // is stored; the first step (beta = -1) yields the seed, in y
            if (cnt < LEG_CHUNK)
                for (int i = cnt + (int)lane; i < LEG_CHUNK; i += 32)
                    stb[i] = make_double2(0.0, 0.0);
            if (j == 0 && lane == 0)
                stb[0].x = -1.0;
            __syncwarp();
            for (int i0 = 0; i0 < cnt; i0 += RED_ROWS)
            {
                const int n = j * LEG_CHUNK + i0 + (int)lane;
                const bool mine = n < ncol;
                double2 prev = make_double2(0.0, 0.0);
                if (stored && mine)
                    prev = col[n];
#pragma unroll
                for (int i = 0; i < RED_ROWS; i++)
                {
                    const double v = fma(t, x, -(stb[i0 + i].x * y));
                    y = x;
                    x = v;
                    red[i * RED_LD + lane] =
                        i & 1 ? make_double2(v * pa.ao, v * pa.bo)
                              : make_double2(v * pa.ae, v * pa.be);
                }
                __syncwarp();
                const double2 tot = row_total(red, lane);
                __syncwarp();
                if (mine)
                    col[n] = make_double2(prev.x + tot.x, prev.y + tot.y);
            }
            if (any_scaled)
            {
                if (leg_fixup(x, y, E))
                    pa = load_amp(A, p, m);
                any_scaled = __any_sync(0xffffffffu, E != 0);
            }
            __syncwarp();
            if (j + 2 < nchunks)
            {
                fence_proxy_async_smem();
                issue(j + 2, s);
            }
        }
        stored = true;
    }
    if (!stored)
        for (int n = (int)lane; n < ncol; n += 32)
            col[n] = make_double2(0.0, 0.0);
    return true;
}

// resident blocks per SM at which each tile width stays free of spills
constexpr int sha_two_min_blocks(int K) { return K >= 8 ? 2 : 3; }

} // namespace

template <int K>
__global__ void __launch_bounds__(128, sha_two_min_blocks(K))
    k_sha_two(const __grid_constant__ ShaTwoArgs A)
{
    extern __shared__ __align__(128) unsigned char smem_raw[];
    const unsigned lane = threadIdx.x & 31u;
    const unsigned warp = threadIdx.x >> 5;
    unsigned char *wbase = smem_raw + (size_t)warp * SHA_WARP_SMEM;
    uint64_t *bar = reinterpret_cast<uint64_t *>(wbase + 2 * SHA_STAGE);
    double2 *red = reinterpret_cast<double2 *>(wbase + 2 * SHA_STAGE + 16);
    auto stg = [&](int s) {
        return reinterpret_cast<double2 *>(wbase + (size_t)s * SHA_STAGE);
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
    const long long TL = two_sum(N);
    const int np = A.npairs;
    const unsigned per = (unsigned)(A.ngroups + (A.nnear > 0 ? 1 : 0));
    bool failed = false;

    for (;;)
    {
        unsigned long long item = 0;
        if (lane == 0)
            item = atomicAdd(A.counter, 1ull);
        item = __shfl_sync(0xffffffffu, item, 0);
        if (item >= (unsigned long long)A.nitems)
            break;
        const long long m = A.m0 + (long long)((unsigned)item / per);
        int sub = (int)((unsigned)item % per);
        if (A.nnear > 0)
        {
            if (sub == 0)
            {
                if (!near_column(A, m, wbase, bar, red, phases))
                    break;
                continue;
            }
            sub--;
        }
        const int g = A.group0 + sub;
        const long long c0 = two_col0(N, m);
        const int nl = (int)two_len(N, m);
        const int nchunks = (nl + TWO_CHUNK - 1) / TWO_CHUNK;
        double2 *col = A.part + 2 * ((size_t)g * (size_t)TL + c0);
        const int tile0 = g * A.tiles_per_group;
        const int tile1 = min(tile0 + A.tiles_per_group, A.ntiles);
        const double sigma = A.sm[m];
        bool stored = false;

        for (int tile = tile0; tile < tile1 && !failed; tile++)
        {
            double z[K], x[K], y[K];
            int E[K];
            PairAmp pa[K];
            bool skip = A.polar_thr >= 0.0;
            bool any_scaled = false, any_live = false;
            auto amp = [&](int k, bool on) {
                const int p = tile * (32 * K) + k * 32 + (int)lane;
                pa[k] = PairAmp{0.0, 0.0, 0.0, 0.0};
                if (on)
                {
                    pa[k] = load_amp(A, p, m);
                    const double t = A.t[p];
                    pa[k].ao *= t;
                    pa[k].bo *= t;
                }
            };
#pragma unroll
            for (int k = 0; k < K; k++)
            {
                const int p = tile * (32 * K) + k * 32 + (int)lane;
                const bool valid = p < np;
                z[k] = valid ? A.z[p] : 0.0;
                x[k] = y[k] = 0.0;
                E[k] = 0;
                if (valid)
                {
                    two_seed(A.pw, A.pw_ld, p, m, sigma, x[k], E[k]);
                    if (!((double)m - (double)N * A.u[p] > A.polar_thr))
                        skip = false;
                }
                // scaled latitudes contribute nothing until they switch
                amp(k, valid && E[k] == 0);
                any_scaled |= E[k] != 0;
                any_live |= E[k] == 0 && x[k] != 0.0;
            }
            if (__all_sync(0xffffffffu, skip))
                continue;
            any_scaled = __any_sync(0xffffffffu, any_scaled);
            any_live = __any_sync(0xffffffffu, any_live);
            const int g0 = tile * (32 * K);
            const bool mixed = g0 < A.polar && g0 + 32 * K > A.polar;
            const double2 *tab = g0 + 32 * K <= A.polar ? A.ag : A.ab;
            auto issue = [&](int j, int s) {
                if (lane == 0)
                {
                    const unsigned bytes =
                        (unsigned)(min(nl - j * TWO_CHUNK, TWO_CHUNK) *
                                   sizeof(double2));
                    mbar_arrive_expect_tx(&bar[s], bytes);
                    bulk_g2s(stg(s), tab + c0 + (long long)j * TWO_CHUNK,
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
                if (!mbar_wait_bounded(&bar[s], (phases >> s) & 1u, A.status))
                {
                    failed = true;
                    break;
                }
                phases ^= 1u << s;
                const int cnt = min(nl - j * TWO_CHUNK, TWO_CHUNK);
                double2 *sab = stg(s);
                // steps beyond the column are formed (from alpha = beta = 0)
                // and not stored
                if (cnt < TWO_CHUNK)
                {
                    if ((int)lane >= cnt)
                        sab[lane] = make_double2(0.0, 0.0);
                    __syncwarp();
                }
                auto advance = [&](int i, auto mix) {
                    const double2 ab = sab[i];
                    const double h = ab.x + ab.y;
#pragma unroll
                    for (int k = 0; k < K; k++)
                    {
                        const double f = fma(
                            ab.x, z[k],
                            decltype(mix)::value && g0 + 32 * k < A.polar
                                ? h : ab.y);
                        const double xn = fma(f, x[k], -y[k]);
                        y[k] = x[k];
                        x[k] = xn;
                    }
                };
                if (any_live)
                {
#pragma unroll 1
                    for (int i0 = 0; i0 < cnt; i0 += RED_ROWS / 2)
                    {
                        // row 2 (step - step0) + parity
                        const long long l =
                            (long long)j * TWO_CHUNK + i0 + (lane >> 1);
                        double2 *cell = col + 2 * l + (lane & 1);
                        const bool mine = l < nl;
                        double2 prev = make_double2(0.0, 0.0);
                        if (stored && mine)
                            prev = *cell;
                        double2 *redl = red + lane;
                        // two steps at a time: eight independent chains of
                        // sums over the pairs (with four, the chains'
                        // latency showed: `wait` stalls first)
                        auto steps = [&](auto mix) {
                            constexpr int U = decltype(mix)::value ? 1 : 4;
#pragma unroll U
                            for (int i = 0; i < RED_ROWS / 2; i += 2)
                            {
                                advance(i0 + i, mix);
                                double ec = 0.0, es = 0.0, oc = 0.0, os = 0.0;
                                double fc = 0.0, fs = 0.0, pc = 0.0, ps = 0.0;
#pragma unroll
                                for (int k = 0; k < K; k++)
                                {
                                    ec = fma(y[k], pa[k].ae, ec);
                                    fc = fma(x[k], pa[k].ae, fc);
                                    es = fma(y[k], pa[k].be, es);
                                    fs = fma(x[k], pa[k].be, fs);
                                    oc = fma(y[k], pa[k].ao, oc);
                                    pc = fma(x[k], pa[k].ao, pc);
                                    os = fma(y[k], pa[k].bo, os);
                                    ps = fma(x[k], pa[k].bo, ps);
                                }
                                advance(i0 + i + 1, mix);
                                redl[0] = make_double2(ec, es);
                                redl[RED_LD] = make_double2(oc, os);
                                redl[2 * RED_LD] = make_double2(fc, fs);
                                redl[3 * RED_LD] = make_double2(pc, ps);
                                redl += 4 * RED_LD;
                            }
                        };
                        if (mixed)
                            steps(std::true_type{});
                        else
                            steps(std::false_type{});
                        __syncwarp();
                        const double2 tot = row_total(red, lane);
                        __syncwarp();
                        if (mine)
                            *cell = make_double2(prev.x + tot.x,
                                                 prev.y + tot.y);
                    }
                }
                else
                {
                    // every latitude below the double range: no sums
                    if (!stored)
                        for (int i = (int)lane; i < 2 * cnt; i += 32)
                            col[2 * j * TWO_CHUNK + i] =
                                make_double2(0.0, 0.0);
                    if (mixed)
                    {
#pragma unroll 2
                        for (int i = 0; i < cnt; i++)
                            advance(i, std::true_type{});
                    }
                    else
                    {
#pragma unroll 4
                        for (int i = 0; i < cnt; i++)
                            advance(i, std::false_type{});
                    }
                }
                if (any_scaled)
                {
                    bool still = false, live = false;
#pragma unroll
                    for (int k = 0; k < K; k++)
                    {
                        if (two_fixup(x[k], y[k], E[k]))
                        {
                            amp(k, true);
                            live = true;
                        }
                        still |= E[k] != 0;
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
            stored = true;
        }
        if (failed)
            break;
        if (!stored)
            for (int i = (int)lane; i < 2 * nl; i += 32)
                col[i] = make_double2(0.0, 0.0);
    }
}

// ---------------------------------------------------------------------------
// C, S of the caller from the groups' partial columns: per order the sums
// Q_l over the groups, even degrees a1_l Q_l + a2_l-1 Q_l-1, odd a3_l Q_l
// (two_tables.cu), plus ct_n times the one-degree column of the equatorial
// pairs (or none), times the degree's rescaling factor (or none); zero above
// nmax.  Memory-bound: the groups are read once.
// ---------------------------------------------------------------------------
__global__ void k_two_reduce(TwoReduceArgs A, long long m_lo)
{
    __shared__ double2 qe[129];
    const long long m = m_lo + blockIdx.x;
    const long long N = A.nmax;
    if (m > A.shc_nmax)
        return;
    const long long d0 = tri_col0(A.shc_nmax, m) - m;
    const long long nl = m <= N ? two_len(N, m) : 0;
    const long long c0 = m <= N ? two_col0(N, m) : 0;
    const long long t0 = m <= N ? tri_col0(N, m) - m : 0;
    const long long TL = two_sum(N);
    const int tid = threadIdx.x;
    if (tid == 0)
        qe[128] = make_double2(0.0, 0.0);
    auto put = [&](long long n, double vc, double vs) {
        if (A.part1)
        {
            const double2 v = A.part1[t0 + n];
            const double k = A.tc[t0 + n];
            vc = fma(k, v.x, vc);
            vs = fma(k, v.y, vs);
        }
        if (A.rescale)
        {
            vc *= A.rescale[n];
            vs *= A.rescale[n];
        }
        A.c[d0 + n] = vc;
        A.s[d0 + n] = vs;
    };
    for (long long l0 = 0; l0 < nl; l0 += 128)
    {
        const long long l = l0 + tid;
        double2 e = make_double2(0.0, 0.0), o = e;
        if (l < nl)
            for (int g = 0; g < A.ngroups; g++)
            {
                const double2 *p = A.part + 2 * ((size_t)g * TL + c0 + l);
                const double2 v = p[0], w = p[1];
                e.x += v.x;
                e.y += v.y;
                o.x += w.x;
                o.y += w.y;
            }
        __syncthreads();
        if (tid == 0)
            qe[0] = qe[128];   // the last of the previous 128 steps
        __syncthreads();
        qe[tid + 1] = e;
        __syncthreads();
        if (l < nl)
        {
            const long long n = m + 2 * l;
            const double a1 = A.kw[c0 + l];
            const double a2 = l > 0 ? A.kw[TL + c0 + l - 1] : 0.0;
            const double a3 = A.kw[2 * TL + c0 + l];
            const double2 q = qe[tid];
            put(n, fma(a1, e.x, a2 * q.x), fma(a1, e.y, a2 * q.y));
            if (n < N)
                put(n + 1, a3 * o.x, a3 * o.y);
        }
    }
    for (long long n = (m <= N ? N + 1 : m) + tid; n <= A.shc_nmax;
         n += blockDim.x)
    {
        A.c[d0 + n] = 0.0;
        A.s[d0 + n] = 0.0;
    }
}

template <int K>
static cudaError_t launch_one(const ShaTwoArgs &A, int grid, cudaStream_t st)
{
    const int warps = 4;
    const size_t smem = (size_t)warps * SHA_WARP_SMEM;
    // beyond the 48 KB default; set once
    static const cudaError_t attr = cudaFuncSetAttribute(
        (const void *)k_sha_two<K>,
        cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (attr != cudaSuccess)
        return attr;
    k_sha_two<K><<<grid, warps * 32, smem, st>>>(A);
    return cudaGetLastError();
}

cudaError_t launch_sha_two(const ShaTwoArgs &A, int K, int grid,
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

cudaError_t launch_two_reduce(const TwoReduceArgs &A, long long m_lo,
                              long long m_hi, cudaStream_t st)
{
    if (m_hi <= m_lo)
        return cudaSuccess;
    k_two_reduce<<<(unsigned)(m_hi - m_lo), 128, 0, st>>>(A, m_lo);
    return cudaGetLastError();
}

} // namespace cb
