// mhh_tdma.cu -- the tridiagonal solves in z of the Poisson equation (Pres_2,
// src/pres_2.cxx:200-326), one column per wave number pair of the x and y
// transforms (mhh_pres.cu).  The default solves keep whole columns in shared
// memory (tdma_mixed_body for the FP32 form, tdma_resident_body for FP64); the
// kernels that sweep through global memory take columns too tall for that and
// the selectable variants.
#include <algorithm>
#include <vector>

#include "mhh_kernels.cuh"
#include "mhh_batchable.cuh"

namespace mhh
{
    // ---------------------------------------------------------------------
    // Tridiagonal solve per spectral column in double, src/pres_2.cxx:200-326:
    // b = dz^2 rho (bmati + bmatj) - (a + c), b[0] += a[0]; the top row gets
    // -c for the mean mode (p = 0 at the top) and +c otherwise (dp/dz = 0);
    // right-hand side dz^2 p; Thomas algorithm.
    //
    // The elimination coefficients depend on the column only through
    // lambda = bmati[i] + bmatj[j], and bmati, bmatj are mirror-symmetric
    // (i and itot - i share a wave number), so the columns form groups of up
    // to four with identical coefficients.  den_k and c_k/den_k of every group
    // are computed once at set-up (k_tdma_table), rounded as the reference
    // rounds them.  The reference-order solve (tdma_body) then repeats the
    // reference's per-cell operations (a product, a difference and a division
    // forward, a product and a difference back) with one thread for the four
    // columns of a group: the mean mode's solve is ill-conditioned, so its
    // result follows every rounding of the sweep.  The rescaled solve
    // (tdma_col_body) needs two FMAs per cell, with one thread per column
    // (tdma_scaled_body: the same with four columns per thread).
    // ---------------------------------------------------------------------
    constexpr double TDMA_FLOAT_GAMMA = 0.999;

    __global__ void k_tdma_table(int niu, int nju, int ktot, const double* __restrict__ bmati,
                                 const double* __restrict__ bmatj, const double* __restrict__ a,
                                 const double* __restrict__ c, const double* __restrict__ dz2rho,
                                 const double* __restrict__ dz2, double* __restrict__ rtab,
                                 double* __restrict__ wtab, double* __restrict__ gtab, double* __restrict__ htab,
                                 float* __restrict__ stab, double* __restrict__ stabd,
                                 unsigned char* __restrict__ fmode)
    {
        const int iu = blockIdx.x*blockDim.x + threadIdx.x;
        const int ju = blockIdx.y;
        if (iu >= niu) return;
        const long long stride = (long long)niu*nju;
        const long long base = iu + (long long)ju*niu;
        const double lam = bmati[iu] + bmatj[ju];
        const bool mean_mode = (iu == 0 && ju == 0);
        // src/pres_2.cxx:266-326 and :200-263, products not contracted.
        double b = mulx(dz2rho[0], lam) - (a[0] + c[0]);
        b += a[0];
        if (ktot == 1) b += mean_mode ? -c[0] : c[0];
        double den = b;
        rtab[base] = den;
        for (int k=1; k<ktot; ++k)
        {
            double bk = mulx(dz2rho[k], lam) - (a[k] + c[k]);
            if (k == ktot-1) bk += mean_mode ? -c[k] : c[k];
            const double w3 = c[k-1]/den;
            wtab[base + (k-1)*stride] = w3;
            den = bk - mulx(a[k], w3);
            rtab[base + k*stride] = den;
        }
        wtab[base + (ktot-1)*stride] = 0.;
        // Rescaled recurrence: with s_k = dz2_k/den_k, y_k = s_k z_k and
        // x_k = s_k xi_k the sweeps become
        //   z_k = p_k - g_k z_{k-1},      g_k = a_k s_{k-1}/dz2_k,
        //   xi_k = z_k - h_k xi_{k+1},    h_k = c_k s_{k+1}/dz2_k,
        // and x_k = s_k xi_k: one FMA per cell and sweep.
        for (int k=0; k<ktot; ++k)
        {
            const double sk = dz2[k]/rtab[base + k*stride];
            if (stabd) stabd[base + k*stride] = sk;
            else stab[base + k*stride] = float(sk);
            gtab[base + k*stride] = k ? a[k]*(dz2[k-1]/rtab[base + (k-1)*stride])/dz2[k] : 0.;
            htab[base + k*stride] = k < ktot-1 ? c[k]*(dz2[k+1]/rtab[base + (k+1)*stride])/dz2[k] : 0.;
        }
        // Float sweeps where the forward sweep damps: a rounding error of z_k
        // enters the next level multiplied by g_{k+1}, and as |g| -> 1 (small
        // |lambda| dz^2: the largest horizontal scales) the forward values
        // become running sums whose round-off grows with the level.  With
        // max |g| <= TDMA_FLOAT_GAMMA the float solve of a column stays
        // within about ten float roundings of its largest value (measured on
        // 256 uniform levels with random right-hand sides: 9 ulp at |g| =
        // 0.999, 4 ulp at 0.9).  The large backward factor h at the top
        // level (the Neumann row) multiplies a value that s scales down, and
        // adds no more.  The groups above the bound and the mean mode keep
        // FP64.
        double gam = 0.;
        for (int k=0; k<ktot; ++k)
            gam = fmax(gam, fabs(gtab[base + k*stride]));
        fmode[base] = (!mean_mode && gam <= TDMA_FLOAT_GAMMA) ? 1 : 0;
    }

    // The k loops run in batches of levels (TDMA_KF forward, TDMA_KBK
    // backward, where the batch holds doubles): the loads of a batch do not
    // depend on the recurrence, so they are issued together and the few
    // threads of this kernel (one per column group) keep enough bytes in
    // flight to stream from HBM instead of waiting one level at a time.
    constexpr int TDMA_KF = 8;
    constexpr int TDMA_KBK = 4;

    // Output of column col at level k.  The mean mode (col 0) is not stored:
    // its level mean (X_00/jtot)/itot goes to dcm[k] and the column gets
    // zero, so that the inverse transforms carry only the other modes and the
    // large hydrostatic part of p stays out of their round-off; the inverse
    // x transform (or the scatter) adds the mean to every point.
    template<typename TF>
    __device__ __forceinline__ TF dc_out(TF val, int col, int k, int itot, int jtot, TF* __restrict__ dcm)
    {
        if (col != 0) return val;
        dcm[k] = TF((double(val) / jtot) / itot);
        return TF(0);
    }

    template<typename TF> struct TdmaP
    {
        int itot, jtot, ktot, niu, nju;
        const double *rtab, *wtab, *a, *dz2, *gtab, *htab;
        const float* stab;
        const double* stabd;
        TF* pk; double* work; TF* dcm;
        const unsigned char* fmode;
        // The column-resident solve: groups per block (log2), coefficients in
        // block order, and the groups with FP64 sweeps.
        int lg, nblk64, nlist;
        const float* ctab; const double* dtab;
        const int* list; const double* ltab; const float* lstab;
    };

    template<typename TF>
    __device__ __forceinline__ void tdma_body(const TdmaP<TF>& A, const VBlock& vb)
    {
        const int itot = A.itot, jtot = A.jtot, ktot = A.ktot, niu = A.niu, nju = A.nju;
        const double* __restrict__ rtab = A.rtab; const double* __restrict__ wtab = A.wtab;
        const double* __restrict__ a = A.a; const double* __restrict__ dz2 = A.dz2;
        TF* __restrict__ pk = A.pk; double* __restrict__ work = A.work; TF* __restrict__ dcm = A.dcm;
        const int iu = vb.x*blockDim.x + threadIdx.x;
        const int ju = vb.y;
        if (iu >= niu) return;
        const long long stride = (long long)niu*nju;
        const long long base = iu + (long long)ju*niu;
        const long long kk = (long long)itot*jtot;
        const int i1 = (iu == 0 || 2*iu == itot) ? -1 : itot - iu;
        const int j1 = (ju == 0 || 2*ju == jtot) ? -1 : jtot - ju;
        // The group's columns (i, j), (itot-i, j), (i, jtot-j), (itot-i, jtot-j);
        // a column that coincides with the first is masked out.  Column
        // offsets within a level are 32-bit (itot*jtot < 2^31 is checked at
        // set-up); level offsets are 64-bit pointers.
        const bool use[4] = {true, i1 >= 0, j1 >= 0, i1 >= 0 && j1 >= 0};
        const int ia = iu, ib = i1 >= 0 ? i1 : iu;
        const int ja = ju*itot, jb = (j1 >= 0 ? j1 : ju)*itot;
        const int col[4] = {ia + ja, ib + ja, ia + jb, ib + jb};

        // Forward sweep: y_k = (dz2_k p_k - a_k y_{k-1}) / den_k, rounded
        // after each operation as in src/pres_2.cxx:200-263.
        double y[4] = {0., 0., 0., 0.};
        for (int k0=0; k0<ktot; k0+=TDMA_KF)
        {
            const int nk = min(TDMA_KF, ktot - k0);
            double r[TDMA_KF];
            TF pv[TDMA_KF][4];
            #pragma unroll
            for (int b=0; b<TDMA_KF; ++b)
            {
                if (b < nk)
                {
                    const long long k = k0 + b;
                    r[b] = __ldg(&rtab[base + k*stride]);
                    const TF* row = pk + k*kk;
                    #pragma unroll
                    for (int q=0; q<4; ++q)
                        if (use[q]) pv[b][q] = row[col[q]];
                }
            }
            #pragma unroll
            for (int b=0; b<TDMA_KF; ++b)
            {
                if (b < nk)
                {
                    const int k = k0 + b;
                    const double dzk = dz2[k];
                    const double ak = a[k];
                    double* wrow = work + (long long)k*kk;
                    #pragma unroll
                    for (int q=0; q<4; ++q)
                    {
                        if (use[q])
                        {
                            double x = mulx(dzk, double(pv[b][q]));
                            if (k) x = x - mulx(ak, y[q]);
                            y[q] = x / r[b];
                            wrow[col[q]] = y[q];
                        }
                    }
                }
            }
        }
        // Back substitution: x_k = y_k - (c_k/den_k) x_{k+1}.
        {
            TF* row = pk + (long long)(ktot-1)*kk;
            #pragma unroll
            for (int q=0; q<4; ++q)
                if (use[q]) row[col[q]] = dc_out<TF>(TF(y[q]), col[q], ktot-1, itot, jtot, dcm);
        }
        for (int k0=ktot-2; k0>=0; k0-=TDMA_KBK)
        {
            const int nk = min(TDMA_KBK, k0 + 1);
            double r[TDMA_KBK];
            double wv[TDMA_KBK][4];
            #pragma unroll
            for (int b=0; b<TDMA_KBK; ++b)
            {
                if (b < nk)
                {
                    const long long k = k0 - b;
                    r[b] = __ldg(&wtab[base + k*stride]);
                    const double* wrow = work + k*kk;
                    #pragma unroll
                    for (int q=0; q<4; ++q)
                        if (use[q]) wv[b][q] = wrow[col[q]];
                }
            }
            #pragma unroll
            for (int b=0; b<TDMA_KBK; ++b)
            {
                if (b < nk)
                {
                    const int k = k0 - b;
                    const double w3 = r[b];
                    TF* row = pk + (long long)k*kk;
                    #pragma unroll
                    for (int q=0; q<4; ++q)
                    {
                        if (use[q])
                        {
                            y[q] = wv[b][q] - mulx(w3, y[q]);
                            row[col[q]] = dc_out<TF>(TF(y[q]), col[q], k, itot, jtot, dcm);
                        }
                    }
                }
            }
        }
    }

    template<typename TF> __device__ __forceinline__ double to_f64(TF v);
    template<> __device__ __forceinline__ double to_f64<float>(float v) { return f2d_exact(v); }
    template<> __device__ __forceinline__ double to_f64<double>(double v) { return v; }

    // Output x_k = s_k xi_k in the field precision: in float the product of
    // the rounded factors (the result is stored in float anyway).
    template<typename TF> __device__ __forceinline__ TF scale_out(double xi, float s, double sd);
    template<> __device__ __forceinline__ float scale_out<float>(double xi, float s, double) { return d2f_rn(xi)*s; }
    template<> __device__ __forceinline__ double scale_out<double>(double xi, float, double sd) { return xi*sd; }

    // The Thomas solve with the rescaled recurrence (coefficients from
    // k_tdma_table): in the float form the whole solve costs two FP64 FMAs
    // per cell, the elimination itself staying in double.
    template<typename TF>
    __device__ __forceinline__ void tdma_scaled_body(const TdmaP<TF>& A, const VBlock& vb)
    {
        const int itot = A.itot, jtot = A.jtot, ktot = A.ktot, niu = A.niu, nju = A.nju;
        const double* __restrict__ gtab = A.gtab; const double* __restrict__ htab = A.htab;
        const float* __restrict__ stab = A.stab; const double* __restrict__ stabd = A.stabd;
        TF* __restrict__ pk = A.pk; double* __restrict__ work = A.work; TF* __restrict__ dcm = A.dcm;
        const int iu = vb.x*blockDim.x + threadIdx.x;
        const int ju = vb.y;
        if (iu >= niu) return;
        const long long stride = (long long)niu*nju;
        const long long base = iu + (long long)ju*niu;
        const long long kk = (long long)itot*jtot;
        const int i1 = (iu == 0 || 2*iu == itot) ? -1 : itot - iu;
        const int j1 = (ju == 0 || 2*ju == jtot) ? -1 : jtot - ju;
        const bool use[4] = {true, i1 >= 0, j1 >= 0, i1 >= 0 && j1 >= 0};
        const int ia = iu, ib = i1 >= 0 ? i1 : iu;
        const int ja = ju*itot, jb = (j1 >= 0 ? j1 : ju)*itot;
        const int col[4] = {ia + ja, ib + ja, ia + jb, ib + jb};

        // Forward: z_k = p_k - g_k z_{k-1}.
        double z[4] = {0., 0., 0., 0.};
        for (int k0=0; k0<ktot; k0+=TDMA_KF)
        {
            const int nk = min(TDMA_KF, ktot - k0);
            double g[TDMA_KF];
            TF pv[TDMA_KF][4];
            #pragma unroll
            for (int b=0; b<TDMA_KF; ++b)
            {
                if (b < nk)
                {
                    const long long k = k0 + b;
                    g[b] = __ldg(&gtab[base + k*stride]);
                    const TF* row = pk + k*kk;
                    #pragma unroll
                    for (int q=0; q<4; ++q)
                        if (use[q]) pv[b][q] = row[col[q]];
                }
            }
            #pragma unroll
            for (int b=0; b<TDMA_KF; ++b)
            {
                if (b < nk)
                {
                    double* wrow = work + (long long)(k0 + b)*kk;
                    #pragma unroll
                    for (int q=0; q<4; ++q)
                    {
                        if (use[q])
                        {
                            z[q] = fma(-g[b], z[q], to_f64<TF>(pv[b][q]));
                            wrow[col[q]] = z[q];
                        }
                    }
                }
            }
        }
        // Backward: xi_k = z_k - h_k xi_{k+1}; x_k = s_k xi_k.
        {
            const long long k = ktot - 1;
            const float s = sizeof(TF) == 4 ? __ldg(&stab[base + k*stride]) : 0.f;
            const double sd = sizeof(TF) == 8 ? __ldg(&stabd[base + k*stride]) : 0.;
            TF* row = pk + k*kk;
            #pragma unroll
            for (int q=0; q<4; ++q)
                if (use[q]) row[col[q]] = dc_out<TF>(scale_out<TF>(z[q], s, sd), col[q], (int)k, itot, jtot, dcm);
        }
        for (int k0=ktot-2; k0>=0; k0-=TDMA_KBK)
        {
            const int nk = min(TDMA_KBK, k0 + 1);
            double h[TDMA_KBK], sd[TDMA_KBK];
            float s[TDMA_KBK];
            double zv[TDMA_KBK][4];
            #pragma unroll
            for (int b=0; b<TDMA_KBK; ++b)
            {
                if (b < nk)
                {
                    const long long k = k0 - b;
                    h[b] = __ldg(&htab[base + k*stride]);
                    s[b] = sizeof(TF) == 4 ? __ldg(&stab[base + k*stride]) : 0.f;
                    sd[b] = sizeof(TF) == 8 ? __ldg(&stabd[base + k*stride]) : 0.;
                    const double* wrow = work + k*kk;
                    #pragma unroll
                    for (int q=0; q<4; ++q)
                        if (use[q]) zv[b][q] = wrow[col[q]];
                }
            }
            #pragma unroll
            for (int b=0; b<TDMA_KBK; ++b)
            {
                if (b < nk)
                {
                    TF* row = pk + (long long)(k0 - b)*kk;
                    #pragma unroll
                    for (int q=0; q<4; ++q)
                    {
                        if (use[q])
                        {
                            z[q] = fma(-h[b], z[q], zv[b][q]);
                            row[col[q]] = dc_out<TF>(scale_out<TF>(z[q], s[b], sd[b]), col[q], k0 - b, itot, jtot, dcm);
                        }
                    }
                }
            }
        }
    }

    // The rescaled solve with one column per thread: the four columns that
    // share the coefficients of one eigenvalue (i, itot-i) x (j, jtot-j) sit
    // in four adjacent lanes, which read the same table entries in one
    // transaction.  Four times the threads of tdma_scaled_body, so that the FP64
    // recurrences and the loads of the next levels of other warps overlap.
    constexpr int TDC_KF = 8;
    constexpr int TDC_KB = 4;

    template<typename TF>
    __device__ __forceinline__ void tdma_col_fp64(const TdmaP<TF>& A, int col, long long base);

    // At most 64 registers, so that eight blocks (32 warps) fit on an SM:
    // the loads of one warp's next levels overlap the FP64 recurrences of
    // the others.
    template<typename TF>
    __device__ __forceinline__ void tdma_col_body(const TdmaP<TF>& A, const VBlock& vb)
    {
        const int itot = A.itot, jtot = A.jtot, niu = A.niu;
        const int t = vb.x*blockDim.x + threadIdx.x;
        const int iu = t >> 2, q = t & 3;
        const int ju = vb.y;
        if (iu >= niu) return;
        const int i1 = (iu == 0 || 2*iu == itot) ? -1 : itot - iu;
        const int j1 = (ju == 0 || 2*ju == jtot) ? -1 : jtot - ju;
        // Lane q holds column (q&1 ? itot-i : i, q&2 ? jtot-j : j); a mirror
        // that coincides with the first column has no lane.
        if (((q & 1) && i1 < 0) || ((q & 2) && j1 < 0)) return;
        const int col = ((q & 1) ? i1 : iu) + ((q & 2) ? j1 : ju)*itot;
        tdma_col_fp64<TF>(A, col, iu + (long long)ju*niu);
    }

    // One column's rescaled solve with the elimination in FP64 (forward
    // values in the FP64 work array).
    template<typename TF>
    __device__ __forceinline__ void tdma_col_fp64(const TdmaP<TF>& A, int col, long long base)
    {
        const int itot = A.itot, jtot = A.jtot, ktot = A.ktot;
        const double* __restrict__ gtab = A.gtab; const double* __restrict__ htab = A.htab;
        const float* __restrict__ stab = A.stab; const double* __restrict__ stabd = A.stabd;
        TF* __restrict__ pk = A.pk; double* __restrict__ work = A.work; TF* __restrict__ dcm = A.dcm;
        const long long stride = (long long)A.niu*A.nju;
        const long long kk = (long long)itot*jtot;

        // Forward: z_k = p_k - g_k z_{k-1}.
        double z = 0.;
        for (int k0=0; k0<ktot; k0+=TDC_KF)
        {
            const int nk = min(TDC_KF, ktot - k0);
            double g[TDC_KF];
            TF pv[TDC_KF];
            #pragma unroll
            for (int b=0; b<TDC_KF; ++b)
                if (b < nk)
                {
                    g[b] = __ldg(gtab + base + (long long)(k0 + b)*stride);
                    pv[b] = pk[col + (long long)(k0 + b)*kk];
                }
            #pragma unroll
            for (int b=0; b<TDC_KF; ++b)
                if (b < nk)
                {
                    z = fma(-g[b], z, to_f64<TF>(pv[b]));
                    work[col + (long long)(k0 + b)*kk] = z;
                }
        }
        // Backward: xi_k = z_k - h_k xi_{k+1}; x_k = s_k xi_k.
        {
            const long long k = ktot - 1;
            const float s = sizeof(TF) == 4 ? __ldg(stab + base + k*stride) : 0.f;
            const double sd = sizeof(TF) == 8 ? __ldg(stabd + base + k*stride) : 0.;
            pk[col + k*kk] = dc_out<TF>(scale_out<TF>(z, s, sd), col, (int)k, itot, jtot, dcm);
        }
        for (int k0=ktot-2; k0>=0; k0-=TDC_KB)
        {
            const int nk = min(TDC_KB, k0 + 1);
            double h[TDC_KB], sd[TDC_KB], zv[TDC_KB];
            float s[TDC_KB];
            #pragma unroll
            for (int b=0; b<TDC_KB; ++b)
                if (b < nk)
                {
                    const long long k = k0 - b;
                    h[b] = __ldg(htab + base + k*stride);
                    s[b] = sizeof(TF) == 4 ? __ldg(stab + base + k*stride) : 0.f;
                    sd[b] = sizeof(TF) == 8 ? __ldg(stabd + base + k*stride) : 0.;
                    zv[b] = work[col + k*kk];
                }
            #pragma unroll
            for (int b=0; b<TDC_KB; ++b)
                if (b < nk)
                {
                    z = fma(-h[b], z, zv[b]);
                    pk[col + (long long)(k0 - b)*kk] = dc_out<TF>(scale_out<TF>(z, s[b], sd[b]), col, k0 - b, itot, jtot, dcm);
                }
        }
    }

    // ---- column-resident solve --------------------------------------------
    // A block keeps whole columns in shared memory: it loads every level of
    // its columns and of their coefficients at once, sweeps forward and back
    // on chip, and stores the solution.  The recurrences are serial in k, so
    // a sweep that loads its levels from global memory waits once per batch
    // of levels; here the loads of a column overlap each other, a level costs
    // about ten cycles of shared-memory and FMA latency, and what bounds the
    // solve is the column loads (scattered 64-byte runs, about half the DRAM
    // rate) and, for short grids, the FP64 chain of the undamped groups (68
    // cycles a level).  Measured per RK3 step (three solves), the sweeps
    // through global memory with batches of sixteen levels against this:
    // FP32 512 x 512 x 256 1.19 -> 0.71 ms, 256 x 256 x 128 0.54 -> 0.089,
    // 150^3 0.617 -> 0.086, 32^3 0.123 -> 0.031; channel 256 x 192 x 128 0.45
    // -> 0.144; FP64 256 x 256 x 128 1.51 -> 0.91, 64^3 0.44 -> 0.080.
    //
    // Columns come in groups of up to four with the same coefficients (see
    // k_tdma_table).  A block owns G = 2^lg consecutive groups, column
    // c = q G + gl being member q of group gl: a warp reads runs of G
    // adjacent cells.  The coefficients of a block are contiguous
    // (k_tdma_chunks): [block][3][ktot][G].
    constexpr int TDR_NT = 256;
    constexpr size_t TDR_SMEM_2 = 113*1024;   // two blocks per SM
    constexpr size_t TDR_SMEM_1 = 224*1024;   // one block per SM

    // Shared memory of a block of G groups: per group and level four columns
    // and three coefficients, all in float or all in double; the FP64 blocks
    // of the mixed solve hold G/2 groups (doubles, the output scale in float).
    inline size_t tdr_smem(int lg, int ktot, bool dbl)
    {
        const size_t kg = (size_t)ktot << lg;
        if (dbl) return 56*kg + 16*(size_t)ktot;
        const size_t kd = (size_t)ktot << (lg ? lg - 1 : 0);
        return std::max(28*kg, 52*kd);
    }

    // log2 of the groups per block, or -1 where not even one group's columns
    // fit: above 4411 levels in the mixed solve (52 bytes a level, those of its
    // FP64 blocks) and 3185 in double (72).  The kernels that sweep through
    // global memory take those.  16
    // groups in float (64-byte runs; the FP64 blocks of the mixed solve then
    // fill a warp) and 8 in double, fewer while that leaves no room for a
    // second block on the SM, and 8 where 16 would leave SMs idle.  Measured
    // per step in float, 32 / 16 / 8 / 4 groups: 36 / 32 / 31 / 31 us at 32^3,
    // 98 / 86 / 80 / 81 at 150^3, 168 / 145 / 215 / 375 for the channel at
    // 256 x 192 x 128 (half its groups in FP64).
    inline int tdr_groups(long long ngroups, int ktot, bool dbl)
    {
        int lg = dbl ? 3 : 4;
        while (lg > 0 && tdr_smem(lg, ktot, dbl) > TDR_SMEM_2) --lg;
        if (tdr_smem(lg, ktot, dbl) > TDR_SMEM_1) return -1;
        if (lg > 3 && (ngroups >> lg) < 2*152) --lg;
        return lg;
    }

    // Coefficients in block order: float (g, h, s) for the mixed solve,
    // double (1/den, den, c/den) for the reference order; with a list, the
    // double (g, h) and float s of the listed groups.
    __global__ void k_tdma_chunks(long long ngroups, int ktot, int lg, const double* __restrict__ rtab,
                                  const double* __restrict__ wtab, const double* __restrict__ gtab,
                                  const double* __restrict__ htab, const float* __restrict__ stab,
                                  float* __restrict__ ctab, double* __restrict__ dtab,
                                  const int* __restrict__ list, int nlist, double* __restrict__ ltab,
                                  float* __restrict__ lstab)
    {
        const long long n = blockIdx.x*(long long)blockDim.x + threadIdx.x;
        const int k = blockIdx.y;
        const int G = 1 << lg;
        const long long blk = n >> lg;
        const int gl = (int)(n & (G - 1));
        const long long limit = list ? (long long)nlist : ngroups;
        const long long rounded = (limit + G - 1) >> lg << lg;
        if (n >= rounded) return;
        const long long grp = n < limit ? (list ? (long long)list[n] : n) : -1;
        const long long t = grp + (long long)k*ngroups;
        const long long o = (blk*3*ktot + k)*G + gl, step = (long long)ktot*G;
        if (list)
        {
            const long long od = (blk*2*ktot + k)*G + gl;
            ltab[od] = grp < 0 ? 0. : gtab[t];
            ltab[od + step] = grp < 0 ? 0. : htab[t];
            lstab[(blk*ktot + k)*G + gl] = grp < 0 ? 0.f : stab[t];
        }
        else if (ctab)
        {
            ctab[o] = grp < 0 ? 0.f : float(gtab[t]);
            ctab[o + step] = grp < 0 ? 0.f : float(htab[t]);
            ctab[o + 2*step] = grp < 0 ? 0.f : stab[t];
        }
        else
        {
            dtab[o] = grp < 0 ? 1. : 1./rtab[t];
            dtab[o + step] = grp < 0 ? 1. : rtab[t];
            dtab[o + 2*step] = grp < 0 ? 0. : wtab[t];
        }
    }

    // Offset of column q of group grp within a level, or -1 if the group has
    // no such column.
    __device__ __forceinline__ int tdr_col(int grp, int q, int niu, int itot, int jtot)
    {
        const int ju = grp / niu, iu = grp - ju*niu;
        if (((q & 1) && (iu == 0 || 2*iu == itot)) || ((q & 2) && (ju == 0 || 2*ju == jtot))) return -1;
        return ((q & 1) ? itot - iu : iu) + ((q & 2) ? jtot - ju : ju)*itot;
    }

    // Asynchronous copy of one element.
    template<typename T>
    __device__ __forceinline__ void tdr_copy(T* dst, const T* src)
    {
        asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n"
                     :: "r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src), "n"(sizeof(T)) : "memory");
    }

    __device__ __forceinline__ void tdr_copy16(void* dst, const void* src)
    {
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n"
                     :: "r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
    }

    // n bytes of a block's coefficients (16-byte copies where the run allows).
    __device__ __forceinline__ void tdr_stage(void* dst, const void* src, size_t n)
    {
        char* d = static_cast<char*>(dst);
        const char* s = static_cast<const char*>(src);
        if (((n | (size_t)s | __cvta_generic_to_shared(d)) & 15) == 0)
            for (size_t e = 16*threadIdx.x; e < n; e += 16*TDR_NT) tdr_copy16(d + e, s + e);
        else
            for (size_t e = 4*threadIdx.x; e < n; e += 4*TDR_NT)
                *reinterpret_cast<float*>(d + e) = *reinterpret_cast<const float*>(s + e);
    }

    // One sweep of the rescaled solve in shared memory, in place: z_k = p_k -
    // g_k z_{k-1} over n levels NC elements apart (NC < 0: downward), the
    // coefficients GS apart.  Whole batches read the next batch while the
    // recurrence runs through the current one.
    template<typename T, int NC, int GS>
    __device__ __forceinline__ void tdr_sweep(T* x, const T* coef, int n)
    {
        constexpr int B = 8;
        T z = T(0);
        int k = 0;
        if (n >= B)
        {
            T p[B], g[B];
            #pragma unroll
            for (int b=0; b<B; ++b) { p[b] = x[b*NC]; g[b] = coef[b*GS]; }
            for (; k + 2*B <= n; k += B)
            {
                T pn[B], gn[B];
                #pragma unroll
                for (int b=0; b<B; ++b) { pn[b] = x[(B + b)*NC]; gn[b] = coef[(B + b)*GS]; }
                #pragma unroll
                for (int b=0; b<B; ++b) { z = fma(-g[b], z, p[b]); x[b*NC] = z; }
                #pragma unroll
                for (int b=0; b<B; ++b) { p[b] = pn[b]; g[b] = gn[b]; }
                x += B*NC; coef += B*GS;
            }
            #pragma unroll
            for (int b=0; b<B; ++b) { z = fma(-g[b], z, p[b]); x[b*NC] = z; }
            x += B*NC; coef += B*GS;
            k += B;
        }
        for (; k<n; ++k) { z = fma(-coef[0], z, x[0]); x[0] = z; x += NC; coef += GS; }
    }

    // The mixed solve of the FP32 form: float sweeps for the groups that damp
    // (fmode 1), FP64 sweeps for the listed others, which the first nblk64
    // blocks take (their chains are the longest).  Per column the arithmetic
    // is that of tdma_col_fp64, in float for the float groups.
    template<int LG>
    __device__ __forceinline__ void tdr_float_block(const TdmaP<float>& A, int blk, unsigned char* smem)
    {
        constexpr int G = 1 << LG, NC = 4*G, LS = TDR_NT/NC;
        const int ktot = A.ktot, tid = threadIdx.x;
        const long long kk = (long long)A.itot*A.jtot;
        // The column this thread copies (levels l0, l0 + LS, ...) and, for
        // the first NC threads, sweeps.
        const int c = tid % NC, gl = c % G, l0 = tid / NC;
        const int n = blk*G + gl;
        const bool in = n < A.niu*A.nju && A.fmode[n];
        if (!__syncthreads_or(in)) return;
        const int col = in ? tdr_col(n, c >> LG, A.niu, A.itot, A.jtot) : -1;
        float* x = reinterpret_cast<float*>(smem);
        float* tab = x + ktot*NC;
        tdr_stage(tab, A.ctab + (size_t)blk*3*ktot*G, sizeof(float)*3*(size_t)ktot*G);
        float* pc = A.pk + col + l0*kk;
        if (col >= 0)
        {
            const float* src = pc;
            float* dst = x + tid;
            #pragma unroll 8
            for (int k=l0; k<ktot; k+=LS) { tdr_copy(dst, src); src += LS*kk; dst += TDR_NT; }
        }
        asm volatile("cp.async.wait_all;\n" ::: "memory");
        __syncthreads();
        if (tid < NC && col >= 0)
        {
            tdr_sweep<float, NC, G>(x + c, tab + gl, ktot);
            tdr_sweep<float, -NC, -G>(x + (ktot - 1)*NC + c, tab + (2*ktot - 1)*G + gl, ktot);
        }
        __syncthreads();
        if (col >= 0)
        {
            const float* xs = x + tid;
            const float* ss = tab + (2*ktot + l0)*G + gl;
            #pragma unroll 8
            for (int k=l0; k<ktot; k+=LS) { *pc = *xs * *ss; pc += LS*kk; xs += TDR_NT; ss += LS*G; }
        }
    }

    template<int LG>
    __device__ __forceinline__ void tdr_fp64_block(const TdmaP<float>& A, int blk, unsigned char* smem)
    {
        constexpr int G = 1 << LG, NC = 4*G, LS = TDR_NT/NC;
        const int ktot = A.ktot, tid = threadIdx.x;
        const long long kk = (long long)A.itot*A.jtot;
        const int c = tid % NC, gl = c % G, l0 = tid / NC;
        const int n = blk*G + gl;
        const int col = n < A.nlist ? tdr_col(A.list[n], c >> LG, A.niu, A.itot, A.jtot) : -1;
        double* x = reinterpret_cast<double*>(smem);
        double* tab = x + ktot*NC;
        float* s = reinterpret_cast<float*>(tab + 2*ktot*G);
        tdr_stage(tab, A.ltab + (size_t)blk*2*ktot*G, sizeof(double)*2*(size_t)ktot*G);
        tdr_stage(s, A.lstab + (size_t)blk*ktot*G, sizeof(float)*(size_t)ktot*G);
        float* pc = A.pk + col + l0*kk;
        if (col >= 0)
        {
            const float* src = pc;
            double* dst = x + tid;
            #pragma unroll 8
            for (int k=l0; k<ktot; k+=LS) { *dst = f2d_exact(*src); src += LS*kk; dst += TDR_NT; }
        }
        asm volatile("cp.async.wait_all;\n" ::: "memory");
        __syncthreads();
        if (tid < NC && col >= 0)
        {
            tdr_sweep<double, NC, G>(x + c, tab + gl, ktot);
            tdr_sweep<double, -NC, -G>(x + (ktot - 1)*NC + c, tab + (2*ktot - 1)*G + gl, ktot);
        }
        __syncthreads();
        if (col > 0)
            for (int k=l0; k<ktot; k+=LS)
            {
                *pc = d2f_rn(x[k*NC + c])*s[k*G + gl];
                pc += LS*kk;
            }
        // The mean mode (group 0, always in FP64 and listed first): its levels
        // over all threads, since dc_out divides twice in double.
        if (blk == 0)
            for (int k=tid; k<ktot; k+=TDR_NT)
                A.pk[k*kk] = dc_out<float>(d2f_rn(x[k*NC])*s[k*G], 0, k, A.itot, A.jtot, A.dcm);
    }

    template<int LG>
    __device__ __forceinline__ void tdma_mixed_body(const TdmaP<float>& A, const VBlock& vb)
    {
        extern __shared__ __align__(16) unsigned char smem_raw[];
        if (vb.x < A.nblk64) tdr_fp64_block<(LG ? LG - 1 : 0)>(A, vb.x, smem_raw);
        else tdr_float_block<LG>(A, vb.x - A.nblk64, smem_raw);
    }

    // x/d from r = 1/d rounded to nearest: the residual of the first quotient
    // corrects it (Markstein 1990).  Three operations instead of a division's
    // dozen on the narrow FP64 pipe.
    __device__ __forceinline__ double div_by(double x, double d, double r)
    {
        const double q = __dmul_rn(x, r);
        return fma(fma(-q, d, x), r, q);
    }

    // The solve in the reference's operation order (tdma_body) in double.
    template<int LG>
    __device__ __forceinline__ void tdma_resident_body(const TdmaP<double>& A, const VBlock& vb)
    {
        constexpr int G = 1 << LG, NC = 4*G, LS = TDR_NT/NC;
        extern __shared__ __align__(16) unsigned char smem_raw[];
        const int ktot = A.ktot, tid = threadIdx.x;
        const long long kk = (long long)A.itot*A.jtot;
        const int c = tid % NC, gl = c % G, l0 = tid / NC;
        const int n = vb.x*G + gl;
        const int col = n < A.niu*A.nju ? tdr_col(n, c >> LG, A.niu, A.itot, A.jtot) : -1;
        double* x = reinterpret_cast<double*>(smem_raw);
        double* tab = x + ktot*NC;
        double* lev = tab + 3*ktot*G;               // a, dz2
        tdr_stage(tab, A.dtab + (size_t)vb.x*3*ktot*G, sizeof(double)*3*(size_t)ktot*G);
        for (int k=tid; k<ktot; k+=TDR_NT) { lev[k] = A.a[k]; lev[ktot + k] = A.dz2[k]; }
        double* pc = A.pk + col + l0*kk;
        if (col >= 0)
        {
            const double* src = pc;
            double* dst = x + tid;
            #pragma unroll 8
            for (int k=l0; k<ktot; k+=LS) { tdr_copy(dst, src); src += LS*kk; dst += TDR_NT; }
        }
        asm volatile("cp.async.wait_all;\n" ::: "memory");
        __syncthreads();
        if (tid < NC && col >= 0)
        {
            // Forward: y_k = (dz2_k p_k - a_k y_{k-1})/den_k.
            constexpr int B = 4;
            double* xc = x + c;
            const double* r = tab + gl;
            const double* den = r + ktot*G;
            double y = 0.;
            auto level = [&](double p, double ri, double dn, double av, bool first)
            {
                y = div_by(first ? p : p - mulx(av, y), dn, ri);
            };
            int k = 0;
            for (; k + B <= ktot; k += B)
            {
                double p[B], ri[B], dn[B], av[B];
                #pragma unroll
                for (int b=0; b<B; ++b)
                {
                    p[b] = mulx(lev[ktot + k + b], xc[b*NC]); ri[b] = r[b*G]; dn[b] = den[b*G]; av[b] = lev[k + b];
                }
                #pragma unroll
                for (int b=0; b<B; ++b) { level(p[b], ri[b], dn[b], av[b], b == 0 && k == 0); xc[b*NC] = y; }
                xc += B*NC; r += B*G; den += B*G;
            }
            for (; k<ktot; ++k)
            {
                level(mulx(lev[ktot + k], xc[0]), r[0], den[0], lev[k], k == 0);
                xc[0] = y;
                xc += NC; r += G; den += G;
            }
            // div_by turns an infinite quotient into a NaN.  A column with a
            // value that is not finite ends in one (a_k is not zero), and
            // sweeps again from its input with the quotients themselves.
            if (!isfinite(y))
            {
                for (k=0; k<ktot; ++k)
                {
                    const double p = mulx(lev[ktot + k], A.pk[col + k*kk]);
                    y = (k ? p - mulx(lev[k], y) : p)/tab[(ktot + k)*G + gl];
                    x[k*NC + c] = y;
                }
            }
            // Back: x_k = y_k - (c_k/den_k) x_{k+1}.
            const double* w3 = tab + (3*ktot - 2)*G + gl;
            xc = x + (ktot - 2)*NC + c;
            k = ktot - 2;
            for (; k + 1 >= B; k -= B)
            {
                double v[B], w[B];
                #pragma unroll
                for (int b=0; b<B; ++b) { v[b] = xc[-b*NC]; w[b] = w3[-b*G]; }
                #pragma unroll
                for (int b=0; b<B; ++b) { y = v[b] - mulx(w[b], y); xc[-b*NC] = y; }
                xc -= B*NC; w3 -= B*G;
            }
            for (; k>=0; --k) { y = xc[0] - mulx(w3[0], y); xc[0] = y; xc -= NC; w3 -= G; }
        }
        __syncthreads();
        if (col > 0)
        {
            const double* xs = x + tid;
            #pragma unroll 8
            for (int k=l0; k<ktot; k+=LS) { *pc = *xs; pc += LS*kk; xs += TDR_NT; }
        }
        // The mean mode's levels over all threads (two divisions each).
        if (vb.x == 0)
            for (int k=tid; k<ktot; k+=TDR_NT) A.pk[k*kk] = dc_out<double>(x[k*NC], 0, k, A.itot, A.jtot, A.dcm);
    }

    // Launches the body for the groups per block that set-up chose.
    template<int LG>
    static void launch_mixed(int lg, unsigned nblk, size_t smem, cudaStream_t s, const TdmaP<float>& A)
    {
        if (lg < LG)
        {
            if constexpr (LG > 0) launch_mixed<LG - 1>(lg, nblk, smem, s, A);
            return;
        }
        set_smem_limit<TdmaP<float>, tdma_mixed_body<LG>, TDR_NT, 2>(TDR_SMEM_1);
        launch_body<TdmaP<float>, tdma_mixed_body<LG>, TDR_NT, 2>(dim3(nblk), dim3(TDR_NT), smem, s, A);
    }

    template<int LG>
    static void launch_resident(int lg, unsigned nblk, size_t smem, cudaStream_t s, const TdmaP<double>& A)
    {
        if (lg < LG)
        {
            if constexpr (LG > 0) launch_resident<LG - 1>(lg, nblk, smem, s, A);
            return;
        }
        set_smem_limit<TdmaP<double>, tdma_resident_body<LG>, TDR_NT, 2>(TDR_SMEM_1);
        launch_body<TdmaP<double>, tdma_resident_body<LG>, TDR_NT, 2>(dim3(nblk), dim3(TDR_NT), smem, s, A);
    }

    int tdma_table(PresWork& pw, int itot, int jtot, int ktot, int precision, cudaStream_t s)
    {
        pw.niu = itot/2 + 1;
        pw.nju = jtot/2 + 1;
        const size_t ng = (size_t)pw.niu*pw.nju, n = ng*ktot;
        const bool dbl = precision == MHH_FP64;
        if (cudaMallocAsync((void**)&pw.rtab, sizeof(double)*n, s) != cudaSuccess) return MHH_ERR_CUDA;
        if (cudaMallocAsync((void**)&pw.wtab, sizeof(double)*n, s) != cudaSuccess) return MHH_ERR_CUDA;
        if (cudaMallocAsync((void**)&pw.gtab, sizeof(double)*n, s) != cudaSuccess) return MHH_ERR_CUDA;
        if (cudaMallocAsync((void**)&pw.htab, sizeof(double)*n, s) != cudaSuccess) return MHH_ERR_CUDA;
        // The output scale in the fields' precision.
        if ((dbl ? cudaMallocAsync((void**)&pw.stabd, sizeof(double)*n, s)
                 : cudaMallocAsync((void**)&pw.stab, sizeof(float)*n, s)) != cudaSuccess) return MHH_ERR_CUDA;
        if (cudaMallocAsync((void**)&pw.fmode, ng, s) != cudaSuccess) return MHH_ERR_CUDA;
        dim3 grid((pw.niu + 127)/128, pw.nju);
        k_tdma_table<<<grid, 128, 0, s>>>(pw.niu, pw.nju, ktot, pw.bmati, pw.bmatj, pw.a, pw.c, pw.dz2rho, pw.dz2,
                                    pw.rtab, pw.wtab, pw.gtab, pw.htab, pw.stab, pw.stabd, pw.fmode);
        count_launch();
        pw.lg = tdr_groups((long long)ng, ktot, dbl);
        if (pw.lg < 0 || ktot > 65535) { pw.lg = -1; return cudaStreamSynchronize(s) == cudaSuccess ? MHH_OK : MHH_ERR_CUDA; }

        // Coefficients in block order.
        auto chunks = [&](int lg, size_t count, const int* list, int nlist)
        {
            const size_t rounded = (count + ((size_t)1 << lg) - 1) >> lg << lg;
            k_tdma_chunks<<<dim3((unsigned)((rounded + 127)/128), ktot), 128, 0, s>>>(
                (long long)ng, ktot, lg, pw.rtab, pw.wtab, pw.gtab, pw.htab, pw.stab, pw.ctab, pw.dtab, list, nlist,
                pw.ltab, pw.lstab);
            count_launch();
        };
        const size_t nr = ((ng + ((size_t)1 << pw.lg) - 1) >> pw.lg << pw.lg)*ktot;
        if ((dbl ? cudaMallocAsync((void**)&pw.dtab, 3*sizeof(double)*nr, s)
                 : cudaMallocAsync((void**)&pw.ctab, 3*sizeof(float)*nr, s)) != cudaSuccess) return MHH_ERR_CUDA;
        chunks(pw.lg, ng, nullptr, 0);
        if (dbl)
        {
            // The resident solve has den and c/den in its blocks' order; no
            // other solve of double fields reads them.
            cudaFreeAsync(pw.rtab, s);
            cudaFreeAsync(pw.wtab, s);
            pw.rtab = pw.wtab = nullptr;
        }
        else
        {
            // The groups with FP64 sweeps, listed on the host.
            std::vector<unsigned char> fm(ng);
            cudaMemcpyAsync(fm.data(), pw.fmode, ng, cudaMemcpyDeviceToHost, s);
            if (cudaStreamSynchronize(s) != cudaSuccess) return MHH_ERR_CUDA;
            std::vector<int> list;
            for (size_t g=0; g<ng; ++g) if (!fm[g]) list.push_back((int)g);
            pw.nlist = (int)list.size();
            const int lgd = pw.lg ? pw.lg - 1 : 0;
            const size_t nl = ((list.size() + ((size_t)1 << lgd) - 1) >> lgd << lgd)*ktot;
            if (cudaMallocAsync((void**)&pw.list, sizeof(int)*list.size(), s) != cudaSuccess) return MHH_ERR_CUDA;
            if (cudaMallocAsync((void**)&pw.ltab, 2*sizeof(double)*nl, s) != cudaSuccess) return MHH_ERR_CUDA;
            if (cudaMallocAsync((void**)&pw.lstab, sizeof(float)*nl, s) != cudaSuccess) return MHH_ERR_CUDA;
            cudaMemcpyAsync(pw.list, list.data(), sizeof(int)*list.size(), cudaMemcpyHostToDevice, s);
            chunks(lgd, list.size(), pw.list, pw.nlist);
            if (cudaStreamSynchronize(s) != cudaSuccess) return MHH_ERR_CUDA;   // list is a host buffer
        }
        return cudaStreamSynchronize(s) == cudaSuccess ? MHH_OK : MHH_ERR_CUDA;
    }

    double tdma_bytes(int itot, int jtot, int ktot, int precision)
    {
        const bool dbl = precision == MHH_FP64;
        const long long ng = (long long)(itot/2 + 1)*(jtot/2 + 1);
        const int lg = ktot > 65535 ? -1 : tdr_groups(ng, ktot, dbl);
        // g, h and the output scale; den and c/den; blocks of the resident
        // solve, in FP32 contexts with every group listed.
        const double each = double(ng)*ktot, blocks = double(((ng + (1LL << std::max(lg, 0)) - 1) >> std::max(lg, 0)) << std::max(lg, 0))*ktot;
        if (dbl) return lg < 0 ? 40.*each : 24.*each + 24.*blocks;
        return 36.*each + double(ng) + (lg < 0 ? 0. : 12.*blocks + 20.*blocks + 4.*ng);
    }

    template<typename TF>
    void launch_tdma(const Dims& d, const PresWork& pw, TF* pk, const KernelOpts& o, cudaStream_t s)
    {
        dim3 grid((pw.niu + 127)/128, pw.nju);
        TF* dcm = static_cast<TF*>(pw.dcm);
        int v = o.tdma < 0 ? (sizeof(TF) == 4 ? 3 : 0) : o.tdma;
        if (v == 3 && (sizeof(TF) == 8 || pw.lg < 0)) v = 1;
        TdmaP<TF> A{d.itot, d.jtot, d.ktot, pw.niu, pw.nju, pw.rtab, pw.wtab, pw.a, pw.dz2, pw.gtab, pw.htab,
                    pw.stab, pw.stabd, pk, pw.work, dcm, pw.fmode, pw.lg, 0, pw.nlist, pw.ctab, pw.dtab, pw.list,
                    pw.ltab, pw.lstab};
        count_launch();
        // The column-resident solves: the mixed one of FP32 contexts and the
        // reference order of FP64 contexts, wherever a group's columns fit in
        // shared memory (lg >= 0).
        const long long ng = (long long)pw.niu*pw.nju;
        const unsigned nblk = pw.lg < 0 ? 0 : (unsigned)((ng + (1 << pw.lg) - 1) >> pw.lg);
        if constexpr (sizeof(TF) == 4)
        {
            if (v == 3)
            {
                const int lgd = pw.lg ? pw.lg - 1 : 0;
                A.nblk64 = (pw.nlist + (1 << lgd) - 1) >> lgd;
                launch_mixed<4>(pw.lg, nblk + A.nblk64, tdr_smem(pw.lg, d.ktot, false), s, A);
                return;
            }
        }
        else if (v == 0 && pw.lg >= 0)
        {
            launch_resident<3>(pw.lg, nblk, tdr_smem(pw.lg, d.ktot, true), s, A);
            return;
        }
        if (v == 1)
        {
            dim3 gridc((4*pw.niu + 127)/128, pw.nju);
            launch_body<TdmaP<TF>, tdma_col_body<TF>, 128, 8>(gridc, dim3(128), 0, s, A);
        }
        else if (v == 2)
            launch_body<TdmaP<TF>, tdma_scaled_body<TF>, 128>(grid, dim3(128), 0, s, A);
        else
            launch_body<TdmaP<TF>, tdma_body<TF>, 128>(grid, dim3(128), 0, s, A);
    }

    template void launch_tdma<float>(const Dims&, const PresWork&, float*, const KernelOpts&, cudaStream_t);
    template void launch_tdma<double>(const Dims&, const PresWork&, double*, const KernelOpts&, cudaStream_t);
}
