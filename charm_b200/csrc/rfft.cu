// Longitude transforms of whole grid rows in shared memory (one CTA, or a
// cluster of CTAs, per row).
//
// CHarm hands every grid row to FFTW: a c2r transform of the lumped
// coefficients in synthesis (src/shs/shs_grd_fft.c) and an r2c transform of
// the row in analysis (src/sha/sha_point.c, FFTW_FORWARD of the real row).
// Grid rows of the quadrature grids have an even length L = 2H whose half
// length H is often not smooth (GL: H = nmax + 1, e.g. 2191 = 7 * 313), so a
// library FFT falls back to slow multi-pass algorithms.  Here one CTA owns a
// row and does everything in shared memory:
//
//   * real <-> complex of half length: z_j = x_2j + i x_2j+1 and
//       X_k = (Z_k + conj Z_H-k)/2 - (i/2) e^(-i pi k/H) (Z_k - conj Z_H-k);
//   * the complex length-H DFT either directly (H = 2^a 3^b) or by
//     Bluestein's chirp-z algorithm (Bluestein 1970): with
//     w_n = exp(-i pi n^2 / H),  DFT(z)_k = w_k sum_j (z_j w_j) conj(w_k-j),
//     a circular convolution of length M >= 2H - 1, M = 2^a 3^b, evaluated
//     as FFT_M, a pointwise product with the precomputed FFT_M of the chirp,
//     and a second FFT_M (conjugated in and out, which inverts it);
//   * FFT_M by in-place Stockham autosort passes (two to four of radix 3 to
//     18 in the compile-time plans, CT_PLANS in rfft.cuh; radix 8, 4, 2 and
//     3 in the run-time plans, which direct transforms, M = 6144 in one CTA,
//     odd rows, the kernel spectra and the clusters without a fixed length
//     use): every thread holds V values
//     across the barrier that separates the loads of a pass from its
//     stores, so one buffer of M values suffices.  The first pass reads its
//     inputs straight from global memory (with the chirp applied; the zero
//     half of the chirped sequence is skipped), and the last pass of the
//     first FFT applies the pointwise product as it stores.  In synthesis
//     the last pass of the second FFT writes the row itself.  Element i
//     lives at i + i/8 in shared memory, which spreads the strided stores
//     of the first pass over the banks;
//   * rows of length 4L whose spectra stop below L (DH2 synthesis): two
//     complex DFTs of length L per row, each computing every other pair of
//     the row (k_rfft_inv4, two CTAs per row);
//   * rows of odd length L (custom grids, synthesis only): one complex DFT
//     of length L by Bluestein, the row being its real part
//     (k_rfft_inv_odd);
//   * transform lengths beyond one CTA's shared memory (M > 9216, e.g. the
//     21602-point rows of the nmax 10800 GL grid, M = 24576): a cluster of
//     C = 2..16 CTAs per row, each holding M / C values, with a radix-C
//     step across the CTAs on either side of the per-CTA FFTs, read
//     through distributed shared memory (k_rfftc_fwd / k_rfftc_inv).
//
// Both directions are unnormalised, as FFTW's and CHarm's: the synthesis
// output is sum_k X_k e^(+2 pi i k n / L) over the Hermitian spectrum, and
// the analysis output is X_k = sum_n x_n e^(-2 pi i k n / L), k <= kmax.
#include "rfft.cuh"

namespace cb
{

// Output of the quarter-length transform: the pair q of half rho of a row
// is the conjugate of DFT value q (w_q conj of the second FFT's output q).
struct OutRowQ
{
    double2 *x2;
    const double2 *w;
    int rho;
    __device__ __forceinline__ void operator()(int q, double2 v) const
    {
        x2[2 * q + rho] = conj2(cmul(__ldg(&w[q]), conj2(v)));
    }
};

// Synthesis of rows of length 4H with spectra below H: CTA 2 row + rho
// computes half rho of the row (SrcQuarter), Bluestein with the plan fixed
// at compile time.
template <int V, int NR, int MC>
__global__ void RFFT_BOUNDS(NR) k_rfft_inv4(RfftArgs A)
{
    extern __shared__ __align__(16) double2 s[];
    const int tid = threadIdx.x;
    const RfftRows R = pick_rows<true>(A);
    const long long row = blockIdx.x >> 1;
    const int rho = (int)(blockIdx.x & 1);
    SrcQuarter src{R.X + row * A.ldX, A.w, A.w4, A.H, R.kmax, rho};
    fft_ct<MC, 0, true>(s, A.tw, tid, src, A.bh);
    fft_ct<MC, 0, false, ct_npass(MC) - 1>(s, A.tw, tid, SrcSmem{s},
                                              nullptr);
    fft_ct_last_out<MC>(
        s, A.tw, tid, A.H,
        OutRowQ{reinterpret_cast<double2 *>(R.x + row * A.ldx), A.w, rho});
}

// Synthesis of rows of odd length L = H: Bluestein over the whole row
// (run-time plan), the row being the real part of the inverse DFT.
template <int V, int NR, bool BATCH>
__global__ void RFFT_BOUNDS(NR) k_rfft_inv_odd(RfftArgs A)
{
    extern __shared__ __align__(16) double2 s[];
    const int tid = threadIdx.x, T = blockDim.x;
    const RfftRows R = pick_rows<BATCH>(A);
    const long long row = blockIdx.x;
    SrcSpectrumOdd src{R.X + row * A.ldX, A.w, A.H, R.kmax};
    dft_h<V, 0>(s, A, tid, T, src);
    double *x = R.x + row * A.ldx;
    for (int j = tid; j < A.H; j += T)
        x[j] = dft_h_out(s, A, j).x;
}

// Analysis direction of a cluster plan (A.C CTAs per row, double rows).
template <int V, int NR, int MC = 0>
__global__ void RFFT_BOUNDS(NR) k_rfftc_fwd(RfftArgs A)
{
    namespace cg = cooperative_groups;
    extern __shared__ __align__(16) double2 s[];
    cg::cluster_group cl = cg::this_cluster();
    const int tid = threadIdx.x, T = blockDim.x;
    const int C = A.C, q = (int)cl.block_rank(), H = A.H;
    const int Mc = A.M / C;
    const long long row = blockIdx.x / C;
    SrcRow src{reinterpret_cast<const double2 *>(A.x + row * A.ldx), A.w, H};
    SrcClusterDif<SrcRow> dif{src, A.twM, q, C, Mc, A.M, H};
    if constexpr (MC > 0)
    {
        // plan fixed at compile time (Mc == MC)
        fft_ct<MC, 0, false>(s, A.tw, tid, dif, A.bh + (size_t)q * Mc);
        fft_ct<MC, 0, false>(s, A.tw, tid, SrcSmem{s}, nullptr);
    }
    else
    {
        fft_m<V>(s, A.tw, Mc, A.npass, tid, T, dif, A.bh + (size_t)q * Mc);
        fft_m<V>(s, A.tw, Mc, A.npass, tid, T, SrcSmem{s}, nullptr);
    }
    cl.sync();
    // this CTA's share of the half spectrum X_0..X_kmax
    const int nk = A.kmax + 1;
    const int k0 = (int)((long long)nk * q / C);
    const int k1 = (int)((long long)nk * (q + 1) / C);
    double2 *X = A.X + row * A.ldX;
    for (int k = k0 + tid; k < k1; k += T)
    {
        const int ka = (k == H) ? 0 : k;
        const int kb = (k == 0) ? 0 : H - k;
        const double2 va = cluster_v(cl, s, A.twM, C, Mc, A.M, ka);
        const double2 vb = cluster_v(cl, s, A.twM, C, Mc, A.M, kb);
        const double2 zk = cmul(__ldg(&A.w[ka]), conj2(va));
        const double2 zh = conj2(cmul(__ldg(&A.w[kb]), conj2(vb)));
        const double2 e = cmul(__ldg(&A.ht[k]), sub2(zk, zh));
        const double2 sm = add2(zk, zh);
        X[k] = make_double2(0.5 * (sm.x + e.y), 0.5 * (sm.y - e.x));
    }
    // no CTA leaves while another still reads its shared memory
    cl.sync();
}

// Synthesis direction of a cluster plan: rows of even length (ODD false,
// pairs x_2t + i x_2t+1 for t < H) or of odd length H (the real part).
template <int V, int NR, bool ODD, int MC, bool BATCH>
__global__ void RFFT_BOUNDS(NR) k_rfftc_inv(RfftArgs A)
{
    namespace cg = cooperative_groups;
    extern __shared__ __align__(16) double2 s[];
    cg::cluster_group cl = cg::this_cluster();
    const int tid = threadIdx.x, T = blockDim.x;
    const int C = A.C, q = (int)cl.block_rank(), H = A.H;
    const int Mc = A.M / C;
    const RfftRows R = pick_rows<BATCH>(A);
    const long long row = blockIdx.x / C;
    if constexpr (ODD)
    {
        SrcSpectrumOdd src{R.X + row * A.ldX, A.w, H, R.kmax};
        SrcClusterDif<SrcSpectrumOdd> dif{src, A.twM, q, C, Mc, A.M, H};
        fft_m<V>(s, A.tw, Mc, A.npass, tid, T, dif, A.bh + (size_t)q * Mc);
    }
    else
    {
        SrcSpectrum src{R.X + row * A.ldX, A.w, A.ht, H, R.kmax};
        SrcClusterDif<SrcSpectrum> dif{src, A.twM, q, C, Mc, A.M, H};
        if constexpr (MC > 0)
            fft_ct<MC, 0, false>(s, A.tw, tid, dif,
                                    A.bh + (size_t)q * Mc);
        else
            fft_m<V>(s, A.tw, Mc, A.npass, tid, T, dif,
                     A.bh + (size_t)q * Mc);
    }
    if constexpr (MC > 0)
        fft_ct<MC, 0, false>(s, A.tw, tid, SrcSmem{s}, nullptr);
    else
        fft_m<V>(s, A.tw, Mc, A.npass, tid, T, SrcSmem{s}, nullptr);
    cl.sync();
    const int t0 = (int)((long long)H * q / C);
    const int t1 = (int)((long long)H * (q + 1) / C);
    for (int t = t0 + tid; t < t1; t += T)
    {
        const double2 v = cluster_v(cl, s, A.twM, C, Mc, A.M, t);
        const double2 z = cmul(__ldg(&A.w[t]), conj2(v));
        if constexpr (ODD)
            R.x[row * A.ldx + t] = z.x;
        else
            reinterpret_cast<double2 *>(R.x + row * A.ldx)[t] = conj2(z);
    }
    cl.sync();
}

// Residue-ordered FFT_M of the Bluestein kernel, times 1/M: CTA q
// (blockIdx.x, no cluster needed) writes bh[q Mc + l] = FFT_M(b)[C l + q] / M.
template <int V, int NR>
__global__ void RFFT_BOUNDS(NR) k_rfftc_kspec(RfftArgs A, double2 *bh)
{
    extern __shared__ __align__(16) double2 s[];
    const int tid = threadIdx.x, T = blockDim.x;
    const int C = A.C, q = (int)blockIdx.x;
    const int Mc = A.M / C;
    SrcClusterDif<SrcKernel> dif{SrcKernel{A.w, A.H, A.M}, A.twM, q, C, Mc,
                                 A.M, A.M};
    fft_m<V>(s, A.tw, Mc, A.npass, tid, T, dif, nullptr);
    const double inv = 1.0 / (double)A.M;
    for (int l = tid; l < Mc; l += T)
    {
        const double2 v = s[pidx(l)];
        bh[(size_t)q * Mc + l] = make_double2(v.x * inv, v.y * inv);
    }
}

// tw[k] = exp(-2 pi i k / n), k < n
__global__ void k_rfft_twiddles(int n, double2 *tw)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n)
    {
        double sn, cs;
        sincospi(2.0 * (double)i / (double)n, &sn, &cs);
        tw[i] = make_double2(cs, -sn);
    }
}

// w4[k] = exp(2 pi i k / 4H), k < H
__global__ void k_rfft_w4(int H, double2 *w4)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < H)
    {
        double sn, cs;
        sincospi((double)k / (2.0 * (double)H), &sn, &cs);
        w4[k] = make_double2(cs, sn);
    }
}

// Tables of one transform length: twiddles exp(-2 pi i k / M), chirp
// w_n = exp(-i pi n^2 / H) (n^2 reduced mod 2H in integers), and
// ht_k = exp(-i pi k / H), k <= H.
__global__ void k_rfft_tables(int H, int M, double2 *tw, double2 *w,
                              double2 *ht)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    double sn, cs;
    if (i < M)
    {
        sincospi(2.0 * (double)i / (double)M, &sn, &cs);
        tw[i] = make_double2(cs, -sn);
    }
    if (w && i < H)
    {
        long long q = ((long long)i * i) % (2LL * H);
        sincospi((double)q / (double)H, &sn, &cs);
        w[i] = make_double2(cs, -sn);
    }
    if (i <= H)
    {
        sincospi((double)i / (double)H, &sn, &cs);
        ht[i] = make_double2(cs, -sn);
    }
}

// FFT_M of the Bluestein kernel, times 1/M.
template <int V, int NR>
__global__ void RFFT_BOUNDS(NR) k_rfft_kernel_spectrum(RfftArgs A, double2 *bh)
{
    extern __shared__ __align__(16) double2 s[];
    const int tid = threadIdx.x, T = blockDim.x;
    fft_m<V>(s, A.tw, A.M, A.npass, tid, T, SrcKernel{A.w, A.H, A.M},
             nullptr);
    const double inv = 1.0 / (double)A.M;
    for (int k = tid; k < A.M; k += T)
    {
        double2 v = s[pidx(k)];
        bh[k] = make_double2(v.x * inv, v.y * inv);
    }
}

size_t rfft_smem_bytes(int M)
{
    return (size_t)(M + M / 8) * sizeof(double2);
}

cudaError_t launch_rfft_tables(RfftArgs &A, double2 *tw, double2 *w,
                               double2 *ht, double2 *bh, cudaStream_t st)
{
    const int n = (A.M > A.H + 1 ? A.M : A.H + 1);
    k_rfft_tables<<<(n + 255) / 256, 256, 0, st>>>(A.H, A.M, tw, w, ht);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess || A.direct)
        return e;
    A.tw = tw;
    A.w = w;
    A.ht = ht;
    const size_t smem = rfft_smem_bytes(A.M);
    k_rfft_kernel_spectrum<16, 96><<<1, A.M / 16, smem, st>>>(A, bh);
    return cudaGetLastError();
}

cudaError_t launch_rfft_w4(int H, double2 *w4, cudaStream_t st)
{
    k_rfft_w4<<<(H + 255) / 256, 256, 0, st>>>(H, w4);
    return cudaGetLastError();
}

cudaError_t rfft_set_smem(size_t smem)
{
    const void *fns[] = {
        (const void *)k_rfft_fwd<false, 0>,
        (const void *)k_rfft_inv<false, 0, false>,
        (const void *)k_rfft_inv<false, 0, true>,
        (const void *)k_rfft_fwd<true, 0>,
        (const void *)k_rfft_inv<true, 0, false>,
        (const void *)k_rfft_inv4<16, 96, 4608>,
        (const void *)k_rfft_kernel_spectrum<16, 96>,
        (const void *)k_rfft_inv_odd<16, 96, false>,
        (const void *)k_rfft_inv_odd<16, 96, true>,
        (const void *)k_rfftc_fwd<16, 96>,
        (const void *)k_rfftc_inv<16, 96, false, 0, false>,
        (const void *)k_rfftc_inv<16, 96, false, 0, true>,
        (const void *)k_rfftc_inv<16, 96, true, 0, false>,
        (const void *)k_rfftc_inv<16, 96, true, 0, true>,
        (const void *)k_rfftc_fwd<16, 96, 6144>,
        (const void *)k_rfftc_inv<16, 96, false, 6144, false>,
        (const void *)k_rfftc_inv<16, 96, false, 6144, true>,
        (const void *)k_rfftc_kspec<16, 96>};
    for (const void *f : fns)
    {
        cudaError_t e = cudaFuncSetAttribute(
            f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess)
            return e;
    }
    // clusters of 16 CTAs (rows beyond 8 x 9216) are a non-portable size
    const void *cfns[] = {(const void *)k_rfftc_fwd<16, 96>,
                          (const void *)k_rfftc_inv<16, 96, false, 0, false>,
                          (const void *)k_rfftc_inv<16, 96, false, 0, true>,
                          (const void *)k_rfftc_inv<16, 96, true, 0, false>,
                          (const void *)k_rfftc_inv<16, 96, true, 0, true>,
                          (const void *)k_rfftc_fwd<16, 96, 6144>,
                          (const void *)k_rfftc_inv<16, 96, false, 6144, false>,
                          (const void *)k_rfftc_inv<16, 96, false, 6144, true>};
    for (const void *f : cfns)
    {
        // where refused, plans with 16 CTAs fail their occupancy check
        // (rfftc_max_clusters) instead
        if (cudaFuncSetAttribute(
                f, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) !=
            cudaSuccess)
            cudaGetLastError();
    }
    return cudaSuccess;
}

int rfftc_max_clusters(int C, int Mc)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)C, 1, 1);
    cfg.blockDim = dim3((unsigned)(Mc / 16), 1, 1);
    cfg.dynamicSmemBytes = rfft_smem_bytes(Mc);
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)C;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, k_rfftc_fwd<16, 96>, &cfg) !=
        cudaSuccess)
    {
        cudaGetLastError();
        return 0;
    }
    int n2 = 0;
    if (cudaOccupancyMaxActiveClusters(
            &n2, k_rfftc_inv<16, 96, false, 0, false>, &cfg) != cudaSuccess)
    {
        cudaGetLastError();
        return 0;
    }
    return n < n2 ? n : n2;
}

cudaError_t launch_rfftc_tables(RfftArgs &A, double2 *tw, double2 *twM,
                                double2 *w, double2 *ht, double2 *bh,
                                cudaStream_t st)
{
    const int Mc = A.M / A.C;
    k_rfft_twiddles<<<(Mc + 255) / 256, 256, 0, st>>>(Mc, tw);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess)
        return e;
    const int n = (A.M > A.H + 1 ? A.M : A.H + 1);
    k_rfft_tables<<<(n + 255) / 256, 256, 0, st>>>(A.H, A.M, twM, w, ht);
    e = cudaGetLastError();
    if (e != cudaSuccess)
        return e;
    A.tw = tw;
    A.twM = twM;
    A.w = w;
    A.ht = ht;
    k_rfftc_kspec<16, 96><<<A.C, Mc / 16, rfft_smem_bytes(Mc), st>>>(A, bh);
    return cudaGetLastError();
}

cudaError_t launch_rfft(const RfftArgs &A, bool inverse, cudaStream_t st)
{
    // the blocks of a batch are the grid's y dimension, 65535 at most
    constexpr int MAX_BATCH = 65535;
    if (A.batch && A.nbatch > MAX_BATCH)
    {
        for (int k = 0; k < A.nbatch; k += MAX_BATCH)
        {
            RfftArgs B = A;
            B.batch = A.batch + k;
            B.nbatch = A.nbatch - k < MAX_BATCH ? A.nbatch - k : MAX_BATCH;
            const cudaError_t e = launch_rfft(B, inverse, st);
            if (e != cudaSuccess)
                return e;
        }
        return cudaSuccess;
    }
    const unsigned grid = (unsigned)A.nrows;
    const unsigned ny = A.batch ? (unsigned)A.nbatch : 1u;
    if (grid == 0 || ny == 0)
        return cudaSuccess;
    if (A.batch && !inverse)
        return cudaErrorInvalidValue;
    if (A.C > 1)
    {
        // one cluster of A.C CTAs per row
        if (A.f32_rows || A.quarter || A.direct || (!inverse && A.odd))
            return cudaErrorInvalidValue;
        const int Mc = A.M / A.C;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(grid * (unsigned)A.C, ny, 1);
        cfg.blockDim = dim3((unsigned)(Mc / 16), 1, 1);
        cfg.dynamicSmemBytes = rfft_smem_bytes(Mc);
        cfg.stream = st;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = (unsigned)A.C;
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        // Mc = 6144 (the nmax 10800 rows): the plan fixed at compile time
        const bool ct = Mc == 6144;
        if (!inverse)
            return ct ? cudaLaunchKernelEx(&cfg, k_rfftc_fwd<16, 96, 6144>, A)
                      : cudaLaunchKernelEx(&cfg, k_rfftc_fwd<16, 96>, A);
        void (*const fn[2][3])(RfftArgs) = {
            {k_rfftc_inv<16, 96, false, 0, false>,
             k_rfftc_inv<16, 96, false, 6144, false>,
             k_rfftc_inv<16, 96, true, 0, false>},
            {k_rfftc_inv<16, 96, false, 0, true>,
             k_rfftc_inv<16, 96, false, 6144, true>,
             k_rfftc_inv<16, 96, true, 0, true>}};
        return cudaLaunchKernelEx(&cfg,
                                  fn[A.batch ? 1 : 0][A.odd ? 2 : ct ? 1 : 0],
                                  A);
    }
    const size_t smem = rfft_smem_bytes(A.M);
    const int T = A.M / 16;
    if (A.odd)
    {
        // rows of odd length: synthesis only, Bluestein, run-time plan
        if (!inverse || A.f32_rows || A.direct)
            return cudaErrorInvalidValue;
        if (A.batch)
            k_rfft_inv_odd<16, 96, true><<<dim3(grid, ny), T, smem, st>>>(A);
        else
            k_rfft_inv_odd<16, 96, false><<<grid, T, smem, st>>>(A);
        return cudaGetLastError();
    }
    if (A.quarter)
    {
        // two CTAs per row (rfft plans set quarter only with M = 4608,
        // double rows, synthesis)
        if (!inverse || A.M != 4608 || A.f32_rows || A.direct)
            return cudaErrorInvalidValue;
        k_rfft_inv4<16, 96, 4608><<<dim3(2 * grid, ny), T, smem, st>>>(A);
        return cudaGetLastError();
    }
    // Bluestein: the plans fixed at compile time, all lengths but 6144
    if (!A.direct)
    {
        static bool (*const group[])(const RfftArgs &, bool, cudaStream_t,
                                     cudaError_t *) = {
            launch_rfft_ct0, launch_rfft_ct1, launch_rfft_ct2,
            launch_rfft_ct3, launch_rfft_ct4, launch_rfft_ct5,
            launch_rfft_ct6};
        cudaError_t e = cudaSuccess;
        for (auto fn : group)
            if (fn(A, inverse, st, &e))
                return e;
    }
    // direct transforms, and the one length (6144) without an even last pass
    const dim3 g2(grid, ny);
    if (A.f32_rows)
    {
        if (A.batch)
            return cudaErrorInvalidValue;
        if (inverse)
            k_rfft_inv<true, 0, false><<<grid, T, smem, st>>>(A);
        else
            k_rfft_fwd<true, 0><<<grid, T, smem, st>>>(A);
    }
    else if (inverse && A.batch)
        k_rfft_inv<false, 0, true><<<g2, T, smem, st>>>(A);
    else if (inverse)
        k_rfft_inv<false, 0, false><<<grid, T, smem, st>>>(A);
    else
        k_rfft_fwd<false, 0><<<grid, T, smem, st>>>(A);
    return cudaGetLastError();
}

} // namespace cb
