// mhh_pres.cu -- the Pres_2 Poisson solve on the GPU without cuFFT:
// divergence of the predicted velocity, hand-written real FFTs along x and y
// (halfcomplex layout, so the spectral solve is the reference's) and the
// scatter back into the ghost-cell layout; the Thomas solve per spectral
// column between the forward and inverse transforms is in mhh_tdma.cu.
//
// FFT: two real sequences x, y of length n are transformed together as
// z = x + i y with a mixed-radix Stockham autosort FFT in shared memory
// (ping-pong buffers, one barrier per stage; run-time plans of radices 2 to 12,
// mhh_fft_plan.h, compile-time stages for n = 32 in float), then separated by
// Hermitian symmetry into FFTW's halfcomplex order r_0 .. r_{n/2}, i_{(n+1)/2-1} .. i_1
// (the convention of src/fft.cxx:145-206).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "mhh_kernels.cuh"
#include "mhh_batchable.cuh"
#include "mhh_fft_plan.h"

namespace mhh
{
    template<typename TF> struct C2;
    template<> struct C2<double> { using T = double2; };
    template<> struct C2<float> { using T = float2; };

    // a + b rounded once and never contracted with a preceding product.
    __device__ __forceinline__ double add_rn(double a, double b) { return __dadd_rn(a, b); }
    __device__ __forceinline__ float add_rn(float a, float b) { return __fadd_rn(a, b); }

    template<typename T2> __device__ __forceinline__ T2 cmul(T2 a, T2 b)
    {
        T2 r; r.x = a.x*b.x - a.y*b.y; r.y = a.x*b.y + a.y*b.x; return r;
    }
    template<typename T2> __device__ __forceinline__ T2 cadd(T2 a, T2 b) { T2 r; r.x = a.x + b.x; r.y = a.y + b.y; return r; }
    template<typename T2> __device__ __forceinline__ T2 csub(T2 a, T2 b) { T2 r; r.x = a.x - b.x; r.y = a.y - b.y; return r; }

    // Packed in float: one instruction per complex sum.
    __device__ __forceinline__ float2 cadd(float2 a, float2 b) { return __fadd2_rn(a, b); }
    __device__ __forceinline__ float2 csub(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.f, -1.f), a); }

    template<typename TF> __device__ __forceinline__ const TF* twtab(const FftPlan& pl);
    template<> __device__ __forceinline__ const double* twtab<double>(const FftPlan& pl) { return pl.tw_d; }
    template<> __device__ __forceinline__ const float* twtab<float>(const FftPlan& pl) { return pl.tw_f; }

    template<typename TF>
    __device__ __forceinline__ typename C2<TF>::T tw(const TF* t, int e)
    {
        typename C2<TF>::T r; r.x = __ldg(t + 2*e); r.y = __ldg(t + 2*e + 1); return r;
    }

    // Quotient and remainder of a / b for 0 <= a < 2^20 and b >= 1 from a
    // float reciprocal rb ~ 1/b: the float quotient is within one of the
    // exact one, and one correction step in either direction makes it exact
    // (a run-time integer division costs several times more).
    __device__ __forceinline__ int div_rcp(int a, int b, float rb, int& rem)
    {
        int q = __float2int_rz(__int2float_rn(a)*rb);
        int r = a - q*b;
        if (r < 0) { --q; r += b; }
        else if (r >= b) { ++q; r -= b; }
        rem = r;
        return q;
    }

    // ---- fixed-length transforms -----------------------------------------
    // The radices are compile-time constants (8 first, then 4), so all index
    // arithmetic folds into shifts and multiplications and each stage is
    // unrolled.
    __host__ __device__ constexpr int fixed_radix(int n, int s)
    {
        return s == 0 && n % 8 == 0 ? 8 : 4;
    }

    template<typename T2>
    __device__ __forceinline__ T2 mul_mi(T2 a) { T2 r; r.x = a.y; r.y = -a.x; return r; }   // -i a

    // Radix-8 DFT (forward, w = exp(-2 pi i/8)) of u[0..7] in place.
    template<typename TF, typename T2>
    __device__ __forceinline__ void dft8(T2* u)
    {
        const TF h = TF(0.70710678118654752440);
        // Stage 1: pairs (q, q+4)
        T2 a0 = cadd(u[0], u[4]), a4 = csub(u[0], u[4]);
        T2 a1 = cadd(u[1], u[5]), a5 = csub(u[1], u[5]);
        T2 a2 = cadd(u[2], u[6]), a6 = csub(u[2], u[6]);
        T2 a3 = cadd(u[3], u[7]), a7 = csub(u[3], u[7]);
        // twiddles w^q on the odd half: a5 *= w, a6 *= w^2 = -i, a7 *= w^3
        T2 t5; t5.x = h*(a5.x + a5.y); t5.y = h*(a5.y - a5.x);
        T2 t6 = mul_mi<T2>(a6);
        T2 t7; t7.x = h*(a7.y - a7.x); t7.y = -h*(a7.x + a7.y);
        // Stage 2: radix-4 on (a0,a1,a2,a3) and (a4,t5,t6,t7)
        T2 b0 = cadd(a0, a2), b2 = csub(a0, a2), b1 = cadd(a1, a3), b3 = mul_mi<T2>(csub(a1, a3));
        T2 c0 = cadd(a4, t6), c2 = csub(a4, t6), c1, c3;
        // By component: the products of t5, t7 are contracted into these sums.
        c1.x = t5.x + t7.x; c1.y = t5.y + t7.y;
        c3.x = t5.y - t7.y; c3.y = -(t5.x - t7.x);
        u[0] = cadd(b0, b1); u[4] = csub(b0, b1);
        u[2] = cadd(b2, b3); u[6] = csub(b2, b3);
        u[1] = cadd(c0, c1); u[5] = csub(c0, c1);
        u[3] = cadd(c2, c3); u[7] = csub(c2, c3);
    }

    // Radix-R butterfly of u[0..R-1] in place (forward).
    template<typename TF, int R>
    __device__ __forceinline__ void radix_bfly(typename C2<TF>::T* u)
    {
        using T2 = typename C2<TF>::T;
        static_assert(R == 8 || R == 4, "radices 8 and 4");
        if (R == 8) dft8<TF, T2>(u);
        else
        {
            const T2 a = cadd(u[0], u[2]), b = csub(u[0], u[2]);
            const T2 c = cadd(u[1], u[3]), e = mul_mi<T2>(csub(u[1], u[3]));
            u[0] = cadd(a, c); u[2] = csub(a, c); u[1] = cadd(b, e); u[3] = csub(b, e);
        }
    }

    // Stockham stages S.. of P sequences of length N, sequence q at src + q*N.
    template<typename TF, int N, int P, int S, int PACC>
    struct FixedStages
    {
        using T2 = typename C2<TF>::T;
        static __device__ __forceinline__ void run(T2*& src, T2*& dst, const T2* __restrict__ tws)
        {
            constexpr int R = fixed_radix(N, S);
            constexpr int T = N / R;
            constexpr int step = N / (PACC*R);
            constexpr int NITEM = P*T;
            for (int it = threadIdx.x; it < NITEM; it += blockDim.x)
            {
                const int seq = it / T;
                const int i = it - seq*T;
                const int k = i % PACC;
                const int xb = seq*N + i;
                const int j = seq*N + (i - k)*R + k;
                T2 u[R];
                u[0] = src[xb];
                #pragma unroll
                for (int q=1; q<R; ++q)
                    u[q] = (PACC == 1) ? src[xb + q*T] : cmul(src[xb + q*T], tws[(q*k*step) % N]);
                radix_bfly<TF, R>(u);
                #pragma unroll
                for (int r=0; r<R; ++r) dst[j + r*PACC] = u[r];
            }
            __syncthreads();
            T2* t = src; src = dst; dst = t;
            FixedStages<TF, N, P, S+1, PACC*R>::run(src, dst, tws);
        }
    };

    template<typename TF, int N, int P, int S>
    struct FixedStages<TF, N, P, S, N>
    {
        using T2 = typename C2<TF>::T;
        static __device__ __forceinline__ void run(T2*&, T2*&, const T2*) {}
    };

    // Right-hand side of the Poisson equation at interior cell (i, j, k)
    // (indices without ghosts), src/pres_2.cxx:155-196: the divergence of the
    // velocity that the tendencies would give after dt.
    template<typename TF>
    __device__ __forceinline__ TF pres_rhs_at(const Dims& d, const Prof<TF>& pr, const TF* __restrict__ u,
                                              const TF* __restrict__ v, const TF* __restrict__ w,
                                              const TF* __restrict__ ut, const TF* __restrict__ vt,
                                              const TF* __restrict__ wt, long long c, int kg, TF dti)
    {
        const long long ii = 1, jj = d.icells, kk = d.ijcells;
        const TF rho = ld(pr.rhoref, kg);
        const TF du = (ld(ut, c+ii) + mulx(ld(u, c+ii), dti)) - (ld(ut, c) + mulx(ld(u, c), dti));
        const TF dv = (ld(vt, c+jj) + mulx(ld(v, c+jj), dti)) - (ld(vt, c) + mulx(ld(v, c), dti));
        const TF dw = mulx(ld(pr.rhorefh, kg+1), ld(wt, c+kk) + mulx(ld(w, c+kk), dti))
                    - mulx(ld(pr.rhorefh, kg  ), ld(wt, c   ) + mulx(ld(w, c   ), dti));
        return mulx(mulx(rho, du), dxi_of<TF>(d)) + mulx(mulx(rho, dv), dyi_of<TF>(d)) + mulx(dw, ld(pr.dzi, kg));
    }

    template<typename TF>
    __device__ __forceinline__ TF pres_rhs(const Dims& d, const Prof<TF>& pr, const TF* __restrict__ u,
                                           const TF* __restrict__ v, const TF* __restrict__ w,
                                           const TF* __restrict__ ut, const TF* __restrict__ vt,
                                           const TF* __restrict__ wt, int i, int j, int k, TF dti)
    {
        return pres_rhs_at(d, pr, u, v, w, ut, vt, wt, ijk(d, i + d.igc, j + d.jgc, k + d.kgc), k + d.kgc, dti);
    }

    // Per-sequence offsets of a tile of nloc <= 16 real sequences starting at
    // s0, computed once per tile by its first threads (the callers
    // synchronise before use): the base of each sequence in data (sb), and
    // for the fused x transforms the ghost-layout offset of the row's first
    // interior cell (sc) and its level k (sk).  Keeps the 64-bit divisions
    // by itot or jtot out of the per-element loops.
    struct TileIdx
    {
        long long sb[16];
        long long sc[16];
        int sk[16];
    };

    // Element j of real sequence s sits at base(s) + j*stride:
    //   rows (x):    base = s*n,                         stride = 1
    //   columns (y): base = (s / itot)*itot*n + s % itot, stride = itot
    struct SeqLayout
    {
        int rows;       // 1: contiguous rows; 0: strided columns
        int itot;       // columns per slab (y layout)
        long long nseq; // number of real sequences
    };

    __device__ __forceinline__ long long seq_base(const SeqLayout& L, long long s, int n)
    {
        if (L.rows) return s*(long long)n;
        // 32-bit division where the sequence number allows (all but the largest
        // grids): a 64-bit one takes longer than a small tile's load.
        const long long k = L.nseq <= 0xffffffffLL ? (long long)((unsigned)s/(unsigned)L.itot) : s/L.itot;
        return k*(long long)L.itot*n + (s - k*L.itot);
    }

    template<typename TF>
    __device__ __forceinline__ void tile_index(TileIdx& ti, const SeqLayout& L, const FftFuse<TF>& fz, long long s0,
                                               int nloc, int n, bool fused)
    {
        const int ls = threadIdx.x;
        if (ls < nloc)
        {
            const long long s = s0 + ls;
            ti.sb[ls] = seq_base(L, s, n);
            if (fused)
            {
                const int kr = (int)(L.nseq <= 0xffffffffLL ? (unsigned)s/(unsigned)fz.d.jtot : s/fz.d.jtot);
                const int jr = (int)(s - (long long)kr*fz.d.jtot);
                ti.sc[ls] = ijk(fz.d, fz.d.igc, jr + fz.d.jgc, kr + fz.d.kgc);
                ti.sk[ls] = kr;
            }
        }
    }

    template<typename TF>
    __device__ __forceinline__ void fft_cp_async(TF* dst, const TF* src, bool valid)
    {
        const unsigned s = (unsigned)__cvta_generic_to_shared(dst);
        const int nb = valid ? (int)sizeof(TF) : 0;
        if constexpr (sizeof(TF) == 4)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" :: "r"(s), "l"(src), "r"(nb) : "memory");
        else
            asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" :: "r"(s), "l"(src), "r"(nb) : "memory");
    }

    // One block transforms 2P real sequences: load them into shared memory,
    // pack pairs as complex, FFT, separate into halfcomplex (forward) or take
    // real and imaginary parts (inverse), store (n = NFIX, P = PFIX).
    // The float transform with the fused right-hand side keeps five blocks
    // per SM (at most 51 registers): its batched loads need the residency to
    // cover the latency of HBM.
    template<typename TF> struct FftP { FftPlan pl; TF* data; SeqLayout L; TF scale; FftFuse<TF> fz; };
    template<typename TF, int FUSE> struct FftOcc { static constexpr int v = (FUSE == 1 && sizeof(TF) == 4) ? 5 : 1; };

    template<typename TF, bool INV, int NFIX, int PFIX, int FUSE>
    __device__ __forceinline__ void fft_body(const FftP<TF>& A, const VBlock& vb)
    {
        const FftPlan& pl = A.pl;
        TF* __restrict__ data = A.data;
        const SeqLayout& L = A.L;
        const TF scale = A.scale;
        const FftFuse<TF>& fz = A.fz;
        using T2 = typename C2<TF>::T;
        extern __shared__ __align__(16) unsigned char smem_raw[];
        constexpr int n = NFIX, P = PFIX;
        // Each buffer holds P complex sequences plus P elements of padding:
        // viewed as 2P real sequences, the column (y) layout strides them by
        // n + 1 so that a warp reading one element of 16+ sequences hits
        // distinct banks.
        T2* buf0 = reinterpret_cast<T2*>(smem_raw);
        T2* buf1 = buf0 + (size_t)P*n + P;
        T2* tws = buf1 + (size_t)P*n + P;  // twiddle table (fixed path)
        const int ns = L.rows ? n : n + 1;  // real-sequence stride in shared memory
        const long long s0 = (long long)vb.x*2*P;
        const int nloc = (int)min((long long)2*P, L.nseq - s0);

        const TF* tt = twtab<TF>(pl);
        for (int e = threadIdx.x; e < n; e += blockDim.x)
        { T2 w; w.x = tt[2*e]; w.y = tt[2*e+1]; tws[e] = w; }

        // 1. Load 2P real sequences into buf1 viewed as real [2P][n], with
        //    asynchronous copies so that all of a thread's loads are in
        //    flight together (a missing sequence reads as zero).
        __shared__ TileIdx ti;
        tile_index<TF>(ti, L, fz, s0, nloc, n, FUSE != 0);
        __syncthreads();
        TF* r1 = reinterpret_cast<TF*>(buf1);
        const int tot = 2*P*n;
        if (FUSE == 1)
        {
            // Rows of the pressure right-hand side computed in place of
            // loading them.  Unrolled so that the loads of several elements
            // are in flight together.
            // RB elements per thread at a time with all their loads issued
            // before the arithmetic (twelve loads each), so that the
            // latency of HBM is covered by the loads of several elements.
            const int kgc = fz.d.kgc;
            constexpr int RB = 4;
            const long long ii = 1, jj = fz.d.icells, kk = fz.d.ijcells;
            for (int e0 = threadIdx.x; e0 < tot; e0 += RB*blockDim.x)
            {
                TF vals[RB][12];
                int kgs[RB];
                #pragma unroll
                for (int b=0; b<RB; ++b)
                {
                    const int e = e0 + b*blockDim.x;
                    const int ls = e / n, i = e - ls*n;
                    const bool ok = e < tot && ls < nloc;
                    // A masked element reads the first interior cell (a valid
                    // address) and is stored as zero below.
                    const long long c = ok ? ti.sc[ls] + i : ti.sc[0];
                    kgs[b] = (ok ? ti.sk[ls] : ti.sk[0]) + kgc;
                    vals[b][0] = ld(fz.ut, c+ii); vals[b][1] = ld(fz.u, c+ii);
                    vals[b][2] = ld(fz.ut, c);    vals[b][3] = ld(fz.u, c);
                    vals[b][4] = ld(fz.vt, c+jj); vals[b][5] = ld(fz.v, c+jj);
                    vals[b][6] = ld(fz.vt, c);    vals[b][7] = ld(fz.v, c);
                    vals[b][8] = ld(fz.wt, c+kk); vals[b][9] = ld(fz.w, c+kk);
                    vals[b][10] = ld(fz.wt, c);   vals[b][11] = ld(fz.w, c);
                }
                #pragma unroll
                for (int b=0; b<RB; ++b)
                {
                    const int e = e0 + b*blockDim.x;
                    if (e < tot)
                    {
                        const int ls = e / n, i = e - ls*n;
                        const TF* x = vals[b];
                        const int kg = kgs[b];
                        const TF rho = ld(fz.pr.rhoref, kg);
                        const TF dti = fz.dti;
                        // The operation order of src/pres_2.cxx:184-191
                        // (products not contracted in double).
                        const TF du = (x[0] + mulx(x[1], dti)) - (x[2] + mulx(x[3], dti));
                        const TF dv = (x[4] + mulx(x[5], dti)) - (x[6] + mulx(x[7], dti));
                        const TF dw = mulx(ld(fz.pr.rhorefh, kg+1), x[8] + mulx(x[9], dti))
                                    - mulx(ld(fz.pr.rhorefh, kg  ), x[10] + mulx(x[11], dti));
                        const TF val = mulx(mulx(rho, du), dxi_of<TF>(fz.d)) + mulx(mulx(rho, dv), dyi_of<TF>(fz.d))
                                     + mulx(dw, ld(fz.pr.dzi, kg));
                        r1[ls*ns + i] = ls < nloc ? val : TF(0);
                    }
                }
            }
        }
        else if (L.rows)
        {
            for (int e = threadIdx.x; e < tot; e += blockDim.x)
            {
                const int ls = e / n, j = e - ls*n;
                const bool ok = ls < nloc;
                fft_cp_async(r1 + ls*ns + j, ok ? data + ti.sb[ls] + j : data, ok);
            }
        }
        else
        {
            // Columns: 2P divides the block size, so every thread keeps
            // one sequence (ls) and walks its elements.
            const int ls = threadIdx.x % (2*P);
            const bool ok = ls < nloc;
            const TF* src = data + (ok ? ti.sb[ls] : 0);
            const long long st = (long long)(blockDim.x/(2*P))*L.itot;
            const TF* sp = src + (long long)(threadIdx.x/(2*P))*L.itot;
            for (int j = threadIdx.x/(2*P); j < n; j += blockDim.x/(2*P), sp += st)
                fft_cp_async(r1 + ls*ns + j, ok ? sp : data, ok);
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
        asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        __syncthreads();

        // 2. Complex input: z = x + i y (forward) or conj(X + i Y) (inverse).
        for (int e = threadIdx.x; e < P*n; e += blockDim.x)
        {
            const int q = e / n, k = e - q*n;
            const TF* hx = r1 + (2*q)*ns;
            const TF* hy = r1 + (2*q+1)*ns;
            T2 z;
            if (!INV)
            {
                z.x = hx[k]; z.y = hy[k];
            }
            else
            {
                const int kk = k <= n/2 ? k : n - k;
                const TF sg = k <= n/2 ? TF(1) : TF(-1);
                const bool real_only = (kk == 0) || (2*kk == n);
                const TF xr = hx[kk], yr = hy[kk];
                const TF xi = real_only ? TF(0) : sg*hx[n - kk];
                const TF yi = real_only ? TF(0) : sg*hy[n - kk];
                z.x = xr - yi;
                z.y = -(xi + yr);
            }
            buf0[e] = z;
        }
        __syncthreads();

        // 3. FFT.
        T2* res = buf0;
        T2* other = buf1;
        FixedStages<TF, NFIX, PFIX, 0, 1>::run(res, other, tws);
        TF* rout = reinterpret_cast<TF*>(other);

        // 4. Real outputs into the other buffer, [2P][n].
        for (int e = threadIdx.x; e < P*n; e += blockDim.x)
        {
            const int q = e / n, k = e - q*n;
            TF* ox = rout + (2*q)*ns;
            TF* oy = rout + (2*q+1)*ns;
            const T2* rq = res + q*n;
            if (!INV)
            {
                if (k <= n/2)
                {
                    const T2 a = rq[k], b = rq[(n - k) % n];
                    const TF xr = TF(0.5)*(a.x + b.x), xi = TF(0.5)*(a.y - b.y);
                    const TF yr = TF(0.5)*(a.y + b.y), yi = TF(-0.5)*(a.x - b.x);
                    ox[k] = xr; oy[k] = yr;
                    if (k > 0 && k < n - k) { ox[n - k] = xi; oy[n - k] = yi; }
                }
            }
            else
            {
                const T2 a = rq[k];
                ox[k] = a.x*scale;
                oy[k] = -a.y*scale;
            }
        }
        __syncthreads();

        // 5. Store (with FUSE == 2 straight into the ghost layout of p, with
        //    the bottom ghost level p[kstart-1] = p[kstart], src/pres_2.cxx:330-358).
        if (FUSE == 2)
        {
            for (int e = threadIdx.x; e < tot; e += blockDim.x)
            {
                const int ls = e / n, i = e - ls*n;
                if (ls < nloc)
                {
                    const TF val = fz.dcm ? add_rn(rout[ls*ns + i], fz.dcm[ti.sk[ls]]) : rout[ls*ns + i];
                    const long long c = ti.sc[ls] + i;
                    fz.p[c] = val;
                    if (ti.sk[ls] == 0) fz.p[c - fz.d.ijcells] = val;
                }
            }
        }
        else if (L.rows)
        {
            for (int e = threadIdx.x; e < tot; e += blockDim.x)
            {
                const int ls = e / n, j = e - ls*n;
                if (ls < nloc) data[ti.sb[ls] + j] = rout[ls*ns + j];
            }
        }
        else
        {
            const int ls = threadIdx.x % (2*P);
            if (ls < nloc)
            {
                const long long st = (long long)(blockDim.x/(2*P))*L.itot;
                TF* dp = data + ti.sb[ls] + (long long)(threadIdx.x/(2*P))*L.itot;
                for (int j = threadIdx.x/(2*P); j < n; j += blockDim.x/(2*P), dp += st)
                    *dp = rout[ls*ns + j];
            }
        }
    }

    template<typename TF, bool INV, int NF, int PF, int FUSE>
    static void launch_fixed(const FftPlan& pl, TF* data, SeqLayout L, TF scale, const FftFuse<TF>& fz, cudaStream_t s)
    {
        const size_t smem = sizeof(typename C2<TF>::T)*((size_t)2*(PF*NF + PF) + NF);
        const long long nblk = (L.nseq + 2*PF - 1) / (2*PF);
        launch_body<FftP<TF>, fft_body<TF, INV, NF, PF, FUSE>, 256, FftOcc<TF, FUSE>::v>(
            dim3((unsigned)nblk), dim3(256), smem, s, FftP<TF>{pl, data, L, scale, fz});
    }

    template<typename TF, bool INV, int NF>
    static bool try_fixed_n(const FftPlan& pl, TF* data, SeqLayout L, TF scale, const FftFuse<TF>& fz, cudaStream_t s)
    {
        if (pl.n != NF) return false;
        // Rows: 4 pairs per block; columns: 4 or 8 (float) pairs per block.
        constexpr int PR = 4, PC = sizeof(TF) == 4 ? 8 : 4;
        if (L.rows)
        {
            if constexpr (!INV) { if (fz.mode == 1) { launch_fixed<TF, INV, NF, PR, 1>(pl, data, L, scale, fz, s); return true; } }
            else { if (fz.mode == 2) { launch_fixed<TF, INV, NF, PR, 2>(pl, data, L, scale, fz, s); return true; } }
            launch_fixed<TF, INV, NF, PR, 0>(pl, data, L, scale, fz, s);
        }
        else if (fft_column_pairs() == 4 || PC == PR) launch_fixed<TF, INV, NF, PR, 0>(pl, data, L, scale, fz, s);
        else launch_fixed<TF, INV, NF, PC, 0>(pl, data, L, scale, fz, s);
        return true;
    }

    // The length with compile-time stages: 32 in float, whose launches are bound
    // by latency and instruction fetches (32^3: 0.088 ms of transforms per step
    // against 0.099 with the run-time plan).  At 16 and from 48 on the run-time
    // plan is as fast or faster, in double at every length.
    template<typename TF, bool INV>
    static bool launch_fixed_any(const FftPlan& pl, TF* data, SeqLayout L, TF scale, const FftFuse<TF>& fz, cudaStream_t s)
    {
        if constexpr (sizeof(TF) == 4) return try_fixed_n<TF, INV, 32>(pl, data, L, scale, fz, s);
        else return false;
    }

    // ---- run-time plans -----------------------------------------------------
    // Any length 2^a 3^b 5^c 7^d.  A block transforms a tile of 2P real
    // sequences (P = 2^lp) held element-major in shared memory, element j of
    // pair q at j*S + q: consecutive threads take the pairs of one element, so
    // the index of a butterfly is a shift, its twiddles are broadcasts, and for
    // columns (y) the pair of adjacent real columns is the complex element as it
    // lies in memory.  Stages of radix 2 to 12 (as few as the length allows) run
    // in registers between two buffers, one barrier each; the first forms the
    // complex input and the store separates the result.  Small tiles, several
    // blocks per SM: what bounds a transform is the latency of its loads and
    // shared-memory stages in float, the FP64 pipe in double.  Transforms in ms
    // per step (x, y), before: one stage per factor with packing and separation
    // passes and two integer divisions per element at 150^3 0.395, 0.313, now
    // 0.193, 0.124; 189 x 105 x 90 0.204, 0.190, now 0.101, 0.104; compile-time
    // stages at 192 (channel 256 x 192 x 128) y 0.181, now 0.156, FP64 1.21, now
    // 1.06; a warp-synchronous schedule at 512 x 512 x 256 2.17, 1.32, now 1.80,
    // 1.31, 256 x 256 x 128 0.333, 0.186, now 0.311, 0.183.  256 threads a block:
    // -3 % at 512, +2 to +15 % at other lengths.
    constexpr int FG_NT = 128;
    constexpr int FG_SMEM = 200*1024;

    template<typename T2> __device__ __forceinline__ void gdft2(T2* u)
    { const T2 a = u[0]; u[0] = cadd(a, u[1]); u[1] = csub(a, u[1]); }

    template<typename TF, typename T2> __device__ __forceinline__ void gdft3(T2& a, T2& b, T2& c)
    {
        const TF s3 = TF(0.86602540378443864676);
        const T2 t1 = cadd(b, c), t4 = csub(b, c);
        T2 t2; t2.x = a.x - TF(0.5)*t1.x; t2.y = a.y - TF(0.5)*t1.y;
        a = cadd(a, t1);
        b.x = t2.x + s3*t4.y; b.y = t2.y - s3*t4.x;
        c.x = t2.x - s3*t4.y; c.y = t2.y + s3*t4.x;
    }

    template<typename T2> __device__ __forceinline__ void gdft4(T2& u0, T2& u1, T2& u2, T2& u3)
    {
        const T2 a = cadd(u0, u2), b = csub(u0, u2), c = cadd(u1, u3), e = mul_mi<T2>(csub(u1, u3));
        u0 = cadd(a, c); u2 = csub(a, c); u1 = cadd(b, e); u3 = csub(b, e);
    }

    // Odd prime R: the pairs u_q, u_{R-q} as sums and differences.
    template<typename TF, typename T2> __device__ __forceinline__ void gdft5(T2& u0, T2& u1, T2& u2, T2& u3, T2& u4)
    {
        const TF c1 = TF(0.30901699437494742410), c2 = TF(-0.80901699437494742410);
        const TF s1 = TF(0.95105651629515357212), s2 = TF(0.58778525229247312917);
        const T2 p1 = cadd(u1, u4), p2 = cadd(u2, u3), m1 = csub(u1, u4), m2 = csub(u2, u3);
        T2 a1, a2, b1, b2;
        a1.x = u0.x + c1*p1.x + c2*p2.x; a1.y = u0.y + c1*p1.y + c2*p2.y;
        a2.x = u0.x + c2*p1.x + c1*p2.x; a2.y = u0.y + c2*p1.y + c1*p2.y;
        b1.x = s1*m1.x + s2*m2.x; b1.y = s1*m1.y + s2*m2.y;
        b2.x = s2*m1.x - s1*m2.x; b2.y = s2*m1.y - s1*m2.y;
        u0 = cadd(u0, cadd(p1, p2));
        u1.x = a1.x + b1.y; u1.y = a1.y - b1.x; u4.x = a1.x - b1.y; u4.y = a1.y + b1.x;
        u2.x = a2.x + b2.y; u2.y = a2.y - b2.x; u3.x = a2.x - b2.y; u3.y = a2.y + b2.x;
    }

    template<typename TF, typename T2> __device__ __forceinline__ void gdft7(T2* u)
    {
        const TF c[3] = {TF(0.62348980185873353053), TF(-0.22252093395631440429), TF(-0.90096886790241912624)};
        const TF s[3] = {TF(0.78183148246802980871), TF(0.97492791218182360702), TF(0.43388373911755812048)};
        T2 p[3], m[3];
        #pragma unroll
        for (int q=0; q<3; ++q) { p[q] = cadd(u[q+1], u[6-q]); m[q] = csub(u[q+1], u[6-q]); }
        const T2 u0 = u[0];
        u[0] = cadd(u0, cadd(p[0], cadd(p[1], p[2])));
        #pragma unroll
        for (int r=1; r<4; ++r)
        {
            T2 a = u0, b; b.x = TF(0); b.y = TF(0);
            #pragma unroll
            for (int q=1; q<4; ++q)
            {
                // cos and sin of 2 pi q r/7 from the first three multiples.
                const int e = (q*r) % 7;
                const TF cc = c[(e < 4 ? e : 7 - e) - 1], ss = e < 4 ? s[e - 1] : -s[6 - e];
                a.x += cc*p[q-1].x; a.y += cc*p[q-1].y;
                b.x += ss*m[q-1].x; b.y += ss*m[q-1].y;
            }
            u[r].x = a.x + b.y; u[r].y = a.y - b.x;
            u[7-r].x = a.x - b.y; u[7-r].y = a.y + b.x;
        }
    }

    // Forward DFT of u[0..R-1] in place.  6 and 10 as 2 x 3 and 2 x 5 by the
    // coprime-factor map (no twiddles), 9 as 3 x 3.
    template<typename TF, int R, typename T2>
    __device__ __forceinline__ void gdft(T2* u)
    {
        if constexpr (R == 2) gdft2(u);
        else if constexpr (R == 3) gdft3<TF>(u[0], u[1], u[2]);
        else if constexpr (R == 4) gdft4(u[0], u[1], u[2], u[3]);
        else if constexpr (R == 5) gdft5<TF>(u[0], u[1], u[2], u[3], u[4]);
        else if constexpr (R == 7) gdft7<TF>(u);
        else if constexpr (R == 8) dft8<TF, T2>(u);
        else if constexpr (R == 6)
        {
            // n = 3 a + 2 b mod 6, k = 3 a' + 4 b' mod 6.
            T2 x[2][3] = {{u[0], u[2], u[4]}, {u[3], u[5], u[1]}};
            gdft3<TF>(x[0][0], x[0][1], x[0][2]);
            gdft3<TF>(x[1][0], x[1][1], x[1][2]);
            #pragma unroll
            for (int b=0; b<3; ++b)
            {
                u[(4*b) % 6] = cadd(x[0][b], x[1][b]);
                u[(4*b + 3) % 6] = csub(x[0][b], x[1][b]);
            }
        }
        else if constexpr (R == 10)
        {
            // n = 5 a + 2 b mod 10, k = 5 a' + 6 b' mod 10.
            T2 x[2][5];
            #pragma unroll
            for (int b=0; b<5; ++b) { x[0][b] = u[2*b]; x[1][b] = u[(2*b + 5) % 10]; }
            gdft5<TF>(x[0][0], x[0][1], x[0][2], x[0][3], x[0][4]);
            gdft5<TF>(x[1][0], x[1][1], x[1][2], x[1][3], x[1][4]);
            #pragma unroll
            for (int b=0; b<5; ++b)
            {
                u[(6*b) % 10] = cadd(x[0][b], x[1][b]);
                u[(6*b + 5) % 10] = csub(x[0][b], x[1][b]);
            }
        }
        else if constexpr (R == 9)
        {
            // X[3 s + r] = sum_a w9^(a r) [DFT3_b u[a + 3 b]](r) w3^(a s).
            const TF c1 = TF(0.76604444311897803520), s1 = TF(-0.64278760968653932632);
            const TF c2 = TF(0.17364817766693034885), s2 = TF(-0.98480775301220805937);
            const TF c4 = TF(-0.93969262078590838405), s4 = TF(-0.34202014332566873304);
            #pragma unroll
            for (int a=0; a<3; ++a) gdft3<TF>(u[a], u[a+3], u[a+6]);
            T2 w1, w2, w4;
            w1.x = c1; w1.y = s1; w2.x = c2; w2.y = s2; w4.x = c4; w4.y = s4;
            u[4] = cmul(u[4], w1); u[5] = cmul(u[5], w2);
            u[7] = cmul(u[7], w2); u[8] = cmul(u[8], w4);
            #pragma unroll
            for (int r=0; r<3; ++r) gdft3<TF>(u[3*r], u[3*r + 1], u[3*r + 2]);
            // u[3 r + s] holds X[3 s + r].
            T2 t;
            t = u[1]; u[1] = u[3]; u[3] = t;
            t = u[2]; u[2] = u[6]; u[6] = t;
            t = u[5]; u[5] = u[7]; u[7] = t;
        }
    }

    template<typename TF> struct FftgP
    {
        TF* data; SeqLayout L; TF scale; FftFuse<TF> fz; const TF* twt;
        int n, lp, nst;
        int pairs;              // columns: the pairs of a tile are adjacent in memory
        unsigned long long fac; // the stages' codes, eight bits each, first stage lowest
    };

    // Complex input element e of a pair: as it lies (forward) or the conjugated
    // halfcomplex pair (inverse).
    template<bool INV, typename T2>
    __device__ __forceinline__ T2 fg_in(const T2* __restrict__ src, int e, int n, int S, int q)
    {
        if (!INV) return src[e*S + q];
        const int kk = 2*e <= n ? e : n - e;
        const bool real_only = kk == 0 || 2*kk == n;
        using TF = std::remove_cv_t<decltype(T2::x)>;
        const T2 a = src[kk*S + q];
        // The imaginary part of a real coefficient is left out, not multiplied
        // by zero: an infinite mean of one row stays out of its partner.
        T2 b; b.x = TF(0); b.y = TF(0);
        if (!real_only) b = src[(n - kk)*S + q];
        const TF sg = 2*e <= n ? TF(1) : TF(-1);
        T2 u;
        u.x = a.x - sg*b.y;
        u.y = -(sg*b.x + a.y);
        return u;
    }

    // One Stockham stage of radix R (p = the product of the radices before):
    // item (i, q), k = i mod p, reads src[i + r T] times w^(r k step) and writes
    // dst[(i - k) R + k + r p].  FIRST: p = 1, no twiddles.
    template<typename TF, int R, bool FIRST, bool INV>
    __device__ __forceinline__ void fg_stage(const typename C2<TF>::T* __restrict__ src, typename C2<TF>::T* __restrict__ dst,
                                             const typename C2<TF>::T* __restrict__ tw, int n, int p, int S, int lp)
    {
        using T2 = typename C2<TF>::T;
        const int T = n/R, step = T/p;
        const float rp = 1.f/(float)p;
        const int q = threadIdx.x & ((1 << lp) - 1);
        for (int i = threadIdx.x >> lp; i < T; i += FG_NT >> lp)
        {
            int k = 0;
            if (!FIRST) div_rcp(i, p, rp, k);
            T2 u[R];
            #pragma unroll
            for (int r=0; r<R; ++r)
            {
                const int e = i + r*T;
                if (FIRST) u[r] = fg_in<INV>(src, e, n, S, q);
                else u[r] = r == 0 ? src[e*S + q] : cmul(src[e*S + q], tw[r*k*step]);
            }
            gdft<TF, R>(u);
            T2* y = dst + ((i - k)*R + k)*S + q;
            #pragma unroll
            for (int r=0; r<R; ++r) y[r*p*S] = u[r];
        }
    }

    // ---- the float plan ------------------------------------------------------
    // In float a transform's rounding shows in every field, so the operations of
    // a length are fixed by its list of elementary radices (plan_floats) and do
    // not depend on how its stages are grouped: two elementary stages RA, RB run
    // in registers as one, with the twiddles of both as if each had been stored.
    //   one stage:  as fg_stage with R = RA;
    //   two:        x[i + r T + q RB T] over q in radix RA (r < RB, twiddles
    //               w^(q k RB step)), then over r in radix RB (m < RA, twiddles
    //               w^(r (k + m p) step)), stored at (i - k) R + k + (m + RA r) p;
    //   RB = 0:     decimation in frequency, the twiddles w^(r (i - k)) on the
    //               results (lengths 128, 256 and 512).
    // Radices 5 and 7 by the direct sum, 8 by dft8.  Sums two at a time in packed
    // instructions, the same roundings: 512 x 512 x 256 x 1.95 ms, now 1.80;
    // 150^3 0.213, 0.138 (x, y), now 0.193, 0.124.
    // The product with its roundings spelled out, so that the sign folded into
    // an operand cannot change which product is contracted.
    __device__ __forceinline__ float2 fe_mul(float2 a, float2 b)
    {
        return make_float2(__fmaf_rn(a.x, b.x, -__fmul_rn(a.y, b.y)), __fmaf_rn(a.y, b.x, __fmul_rn(a.x, b.y)));
    }

    template<int R>
    __device__ __forceinline__ void fe_dft(float2* u, const float2* __restrict__ tw, int n)
    {
        if constexpr (R == 2) gdft2(u);
        else if constexpr (R == 3) gdft3<float>(u[0], u[1], u[2]);
        else if constexpr (R == 4) gdft4(u[0], u[1], u[2], u[3]);
        else if constexpr (R == 8) dft8<float, float2>(u);
        else
        {
            // Packed: (x, y) of u_q w = (u.x, u.y) (w.x, w.x) + (u.y, u.x) (-w.y, w.y).
            float2 wx[R], wy[R], v[R];
            #pragma unroll
            for (int m=0; m<R; ++m)
            {
                const float2 w = tw[m*(n/R)];
                wx[m] = make_float2(w.x, w.x);
                wy[m] = make_float2(-w.y, w.y);
            }
            #pragma unroll
            for (int r=0; r<R; ++r) v[r] = u[0];
            #pragma unroll
            for (int q=1; q<R; ++q)
            {
                const float2 t = make_float2(u[q].y, u[q].x);
                #pragma unroll
                for (int r=0; r<R; ++r)
                    v[r] = __fadd2_rn(v[r], __ffma2_rn(u[q], wx[(q*r) % R], __fmul2_rn(t, wy[(q*r) % R])));
            }
            #pragma unroll
            for (int r=0; r<R; ++r) u[r] = v[r];
        }
    }

    template<int RA, int RB, bool FIRST, bool INV>
    __device__ __forceinline__ void fe_stage(const float2* __restrict__ src, float2* __restrict__ dst,
                                             const float2* __restrict__ tw, int n, int p, int S, int lp)
    {
        constexpr bool DIF = RB == 0;
        constexpr int B = RB > 1 ? RB : 1, R = RA*B;
        const int T = n/R, step = T/p;
        const float rp = 1.f/(float)p;
        const int q = threadIdx.x & ((1 << lp) - 1);
        for (int i = threadIdx.x >> lp; i < T; i += FG_NT >> lp)
        {
            int k = 0;
            if (!FIRST) div_rcp(i, p, rp, k);
            float2 u[B][RA];
            #pragma unroll
            for (int r=0; r<B; ++r)
            {
                #pragma unroll
                for (int a=0; a<RA; ++a)
                {
                    const int e = i + (r + a*B)*T;
                    if (FIRST) u[r][a] = fg_in<INV>(src, e, n, S, q);
                    else u[r][a] = DIF || a == 0 ? src[e*S + q] : fe_mul(src[e*S + q], tw[a*k*B*step]);
                }
                fe_dft<RA>(u[r], tw, n);
            }
            float2* y = dst + ((i - k)*R + k)*S + q;
            if (DIF)
            {
                if (p != T)
                {
                    #pragma unroll
                    for (int a=1; a<RA; ++a) u[0][a] = fe_mul(u[0][a], tw[a*(i - k)]);
                }
                #pragma unroll
                for (int a=0; a<RA; ++a) y[a*p*S] = u[0][a];
            }
            else
            {
                #pragma unroll
                for (int m=0; m<RA; ++m)
                {
                    float2 v[B];
                    v[0] = u[0][m];
                    #pragma unroll
                    for (int r=1; r<B; ++r) v[r] = FIRST && m == 0 ? u[r][m] : fe_mul(u[r][m], tw[r*(k + m*p)*step]);
                    if constexpr (B > 1) fe_dft<B>(v, tw, n);
                    #pragma unroll
                    for (int r=0; r<B; ++r) y[(m + RA*r)*p*S] = v[r];
                }
            }
        }
    }

    // A stage of the plan: code R in double, RA + 16 RB in float.
    template<typename TF, bool FIRST, bool INV>
    __device__ __forceinline__ void fg_any(int code, const typename C2<TF>::T* src, typename C2<TF>::T* dst,
                                           const typename C2<TF>::T* tw, int n, int p, int S, int lp)
    {
        if constexpr (sizeof(TF) == 8)
            switch (code)
            {
                case 2: fg_stage<TF, 2, FIRST, INV>(src, dst, tw, n, p, S, lp); break;
                case 3: fg_stage<TF, 3, FIRST, INV>(src, dst, tw, n, p, S, lp); break;
                case 4: fg_stage<TF, 4, FIRST, INV>(src, dst, tw, n, p, S, lp); break;
                case 5: fg_stage<TF, 5, FIRST, INV>(src, dst, tw, n, p, S, lp); break;
                case 6: fg_stage<TF, 6, FIRST, INV>(src, dst, tw, n, p, S, lp); break;
                case 7: fg_stage<TF, 7, FIRST, INV>(src, dst, tw, n, p, S, lp); break;
                case 8: fg_stage<TF, 8, FIRST, INV>(src, dst, tw, n, p, S, lp); break;
                case 9: fg_stage<TF, 9, FIRST, INV>(src, dst, tw, n, p, S, lp); break;
                default: fg_stage<TF, 10, FIRST, INV>(src, dst, tw, n, p, S, lp); break;
            }
        else
            switch (code)
            {
                case 0x02: if (FIRST) fe_stage<2, 0, true, INV>(src, dst, tw, n, p, S, lp); break;
                case 0x04: if (FIRST) fe_stage<4, 0, true, INV>(src, dst, tw, n, p, S, lp); break;
                case 0x08: fe_stage<8, 0, FIRST, INV>(src, dst, tw, n, p, S, lp); break;
                case 0x12: fe_stage<2, 1, FIRST, INV>(src, dst, tw, n, p, S, lp); break;
                case 0x13: fe_stage<3, 1, FIRST, INV>(src, dst, tw, n, p, S, lp); break;
                case 0x14: fe_stage<4, 1, FIRST, INV>(src, dst, tw, n, p, S, lp); break;
                case 0x15: fe_stage<5, 1, FIRST, INV>(src, dst, tw, n, p, S, lp); break;
                case 0x17: fe_stage<7, 1, FIRST, INV>(src, dst, tw, n, p, S, lp); break;
                case 0x18: fe_stage<8, 1, FIRST, INV>(src, dst, tw, n, p, S, lp); break;
                case 0x32: fe_stage<2, 3, FIRST, INV>(src, dst, tw, n, p, S, lp); break;
                case 0x52: fe_stage<2, 5, FIRST, INV>(src, dst, tw, n, p, S, lp); break;
                case 0x24: fe_stage<4, 2, FIRST, INV>(src, dst, tw, n, p, S, lp); break;
                case 0x33: fe_stage<3, 3, FIRST, INV>(src, dst, tw, n, p, S, lp); break;
                default:   fe_stage<4, 3, FIRST, INV>(src, dst, tw, n, p, S, lp); break;
            }
    }

    template<typename T2>
    __device__ __forceinline__ void fg_copy2(T2* dst, const T2* src)
    {
        asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n"
                     :: "r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src), "n"(sizeof(T2)) : "memory");
    }

    template<typename TF, bool INV, int FUSE, bool ROWS>
    __device__ __forceinline__ void fftg_body(const FftgP<TF>& A, const VBlock& vb)
    {
        using T2 = typename C2<TF>::T;
        const int n = A.n, lp = A.lp, P = 1 << lp, S = P + (lp ? 1 : 0);
        const SeqLayout& L = A.L;
        const FftFuse<TF>& fz = A.fz;
        extern __shared__ __align__(16) unsigned char smem_raw[];
        T2* b0 = reinterpret_cast<T2*>(smem_raw);
        T2* b1 = b0 + (size_t)n*S;
        T2* tw = b1 + (size_t)n*S;
        __shared__ TileIdx ti;
        const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
        const long long s0 = (long long)vb.x*2*P;
        const int nloc = (int)min((long long)2*P, L.nseq - s0);
        tile_index<TF>(ti, L, fz, s0, nloc, n, FUSE != 0);
        __syncthreads();
        for (int e = tid; e < n; e += FG_NT) fg_copy2(tw + e, reinterpret_cast<const T2*>(A.twt) + e);

        // 1. Load; a missing sequence reads as zero.
        TF* r0 = reinterpret_cast<TF*>(b0);
        if (FUSE == 1)
        {
            // Rows of the pressure right-hand side in place of a load
            // (src/pres_2.cxx:155-196), a warp per row.
            const Dims& d = fz.d;
            for (int ls = warp; ls < 2*P; ls += FG_NT/32)
            {
                TF* dst = r0 + ls;                  // component ls & 1 of pair ls >> 1
                if (ls < nloc)
                {
                    const long long c = ti.sc[ls];
                    const int kg = ti.sk[ls] + d.kgc;
                    const TF rho = ld(fz.pr.rhoref, kg), rb = ld(fz.pr.rhorefh, kg), rt = ld(fz.pr.rhorefh, kg+1);
                    const TF dzi = ld(fz.pr.dzi, kg), dti = fz.dti;
                    const TF *u = fz.u + c, *v = fz.v + c, *w = fz.w + c, *ut = fz.ut + c, *vt = fz.vt + c, *wt = fz.wt + c;
                    const int jj = d.icells, kk = d.ijcells;
                    #pragma unroll 4
                    for (int i = lane; i < n; i += 32)
                    {
                        const TF du = (ld(ut, i+1) + mulx(ld(u, i+1), dti)) - (ld(ut, i) + mulx(ld(u, i), dti));
                        const TF dv = (ld(vt, i+jj) + mulx(ld(v, i+jj), dti)) - (ld(vt, i) + mulx(ld(v, i), dti));
                        const TF dw = mulx(rt, ld(wt, i+kk) + mulx(ld(w, i+kk), dti)) - mulx(rb, ld(wt, i) + mulx(ld(w, i), dti));
                        dst[2*i*S] = mulx(mulx(rho, du), dxi_of<TF>(d)) + mulx(mulx(rho, dv), dyi_of<TF>(d)) + mulx(dw, dzi);
                    }
                }
                else
                    for (int i = lane; i < n; i += 32) dst[2*i*S] = TF(0);
            }
        }
        else if (ROWS)
        {
            for (int ls = warp; ls < 2*P; ls += FG_NT/32)
            {
                const bool ok = ls < nloc;
                const TF* src = ok ? A.data + ti.sb[ls] : A.data;
                #pragma unroll 4
                for (int i = lane; i < n; i += 32) fft_cp_async(r0 + ls + 2*i*S, ok ? src + i : src, ok);
            }
        }
        else
        {
            const int q = tid & (P - 1);
            const bool ok0 = 2*q < nloc, ok1 = 2*q + 1 < nloc;
            const TF* x = A.data + (ok0 ? ti.sb[2*q] : 0);
            const TF* y = A.data + (ok1 ? ti.sb[2*q + 1] : 0);
            if (A.pairs && ok1)
            {
                #pragma unroll 4
                for (int j = tid >> lp; j < n; j += FG_NT >> lp)
                    fg_copy2(b0 + j*S + q, reinterpret_cast<const T2*>(x + (long long)j*L.itot));
            }
            else
                for (int j = tid >> lp; j < n; j += FG_NT >> lp)
                {
                    fft_cp_async(r0 + 2*(j*S + q), ok0 ? x + (long long)j*L.itot : x, ok0);
                    fft_cp_async(r0 + 2*(j*S + q) + 1, ok1 ? y + (long long)j*L.itot : y, ok1);
                }
        }
        asm volatile("cp.async.wait_all;\n" ::: "memory");
        __syncthreads();

        // 2. Stages.
        T2* src = b0;
        T2* dst = b1;
        int p = 1;
        for (int st=0; st<A.nst; ++st)
        {
            const int code = (int)(A.fac >> 8*st) & 255;
            if (st == 0) fg_any<TF, true, INV>(code, src, dst, tw, n, 1, S, lp);
            else fg_any<TF, false, INV>(code, src, dst, tw, n, p, S, lp);
            p *= code < 32 ? code & 15 : (code & 15)*(code >> 4);
            __syncthreads();
            T2* t = src; src = dst; dst = t;
        }

        // 3. Store: real and imaginary parts (inverse) or the halfcomplex
        //    separation (forward).
        auto pair_out = [&](int k, int q) -> T2
        {
            T2 o;
            if (INV)
            {
                const T2 a = src[k*S + q];
                o.x = a.x*A.scale; o.y = -a.y*A.scale;
            }
            else
            {
                const int kk = 2*k <= n ? k : n - k;
                const T2 a = src[kk*S + q], b = src[(kk == 0 ? 0 : n - kk)*S + q];
                if (2*k <= n) { o.x = TF(0.5)*(a.x + b.x); o.y = TF(0.5)*(a.y + b.y); }
                else { o.x = TF(0.5)*(a.y - b.y); o.y = TF(-0.5)*(a.x - b.x); }
            }
            return o;
        };
        if (ROWS)
        {
            // A warp (or, with fewer pairs than warps, several) per pair of rows.
            constexpr int NW = FG_NT/32;
            const int wpp = P < NW ? NW/P : 1;
            for (int q = warp/wpp; 2*q < nloc; q += NW/wpp)
            {
                const bool two = 2*q + 1 < nloc;
                if (FUSE == 2)
                {
                    // Straight into the ghost layout of p, with the bottom
                    // ghost level p[kstart-1] = p[kstart]
                    // (src/pres_2.cxx:330-358).
                    const int l0 = 2*q, l1 = two ? 2*q + 1 : 2*q;
                    TF* x = fz.p + ti.sc[l0];
                    TF* y = fz.p + ti.sc[l1];
                    const TF m0 = fz.dcm ? fz.dcm[ti.sk[l0]] : TF(0), m1 = fz.dcm ? fz.dcm[ti.sk[l1]] : TF(0);
                    const bool g0 = ti.sk[l0] == 0, g1 = ti.sk[l1] == 0;
                    #pragma unroll 4
                    for (int i = lane + 32*(warp % wpp); i < n; i += 32*wpp)
                    {
                        T2 o = pair_out(i, q);
                        if (fz.dcm) { o.x = add_rn(o.x, m0); o.y = add_rn(o.y, m1); }
                        x[i] = o.x;
                        if (g0) x[i - fz.d.ijcells] = o.x;
                        if (two)
                        {
                            y[i] = o.y;
                            if (g1) y[i - fz.d.ijcells] = o.y;
                        }
                    }
                }
                else
                {
                    TF* x = A.data + ti.sb[2*q];
                    TF* y = A.data + ti.sb[two ? 2*q + 1 : 2*q];
                    #pragma unroll 4
                    for (int i = lane + 32*(warp % wpp); i < n; i += 32*wpp)
                    {
                        const T2 o = pair_out(i, q);
                        x[i] = o.x;
                        if (two) y[i] = o.y;
                    }
                }
            }
        }
        else
        {
            const int q = tid & (P - 1);
            const bool ok0 = 2*q < nloc, ok1 = 2*q + 1 < nloc;
            TF* x = A.data + (ok0 ? ti.sb[2*q] : 0);
            TF* y = A.data + (ok1 ? ti.sb[2*q + 1] : 0);
            for (int j = tid >> lp; j < n; j += FG_NT >> lp)
            {
                const T2 o = pair_out(j, q);
                const long long e = (long long)j*L.itot;
                if (A.pairs && ok1) *reinterpret_cast<T2*>(x + e) = o;
                else
                {
                    if (ok0) x[e] = o.x;
                    if (ok1) y[e] = o.y;
                }
            }
        }
    }

    template<typename TF, bool INV, int FUSE, bool ROWS>
    static void launch_generic(const FftPlan& pl, TF* data, SeqLayout L, TF scale, const FftFuse<TF>& fz, cudaStream_t s)
    {
        using T2 = typename C2<TF>::T;
        using B = FftgP<TF>;
        constexpr auto body = fftg_body<TF, INV, FUSE, ROWS>;
        B A{};
        A.data = data; A.L = L; A.scale = scale; A.fz = fz;
        A.twt = sizeof(TF) == 8 ? reinterpret_cast<const TF*>(pl.tw_d) : reinterpret_cast<const TF*>(pl.tw_f);
        A.n = pl.n;
        A.nst = sizeof(TF) == 8 ? pl.ngfac : pl.nffac;
        for (int q=0; q<A.nst && q<8; ++q) A.fac |= (unsigned long long)(sizeof(TF) == 8 ? pl.gfac[q] : pl.ffac[q]) << 8*q;
        // Pairs per tile, at most eight: columns as many as leave two (float) or
        // more (double, bound by the FP64 pipe) blocks on an SM, so that a run is
        // 64 bytes or more; rows, which need no runs, few enough that five
        // blocks' loads overlap (512 x 512 x 256, 8, 4, 2
        // pairs: 2.48, 1.85, 2.06 ms per step for x; 150^3 0.177, 0.192, 0.239;
        // with scalar sums).
        auto bytes = [&](int lp) { return sizeof(T2)*(size_t)pl.n*(2*((1 << lp) + (lp ? 1 : 0)) + 1); };
        const size_t most = (ROWS ? 46 : (sizeof(TF) == 4 ? 80 : 48))*1024;
        A.lp = ROWS && sizeof(TF) == 8 ? 2 : 3;
        while (A.lp > 1 && bytes(A.lp) > most) --A.lp;
        if (bytes(A.lp) > (size_t)FG_SMEM) A.lp = 0;
        // Pairs of columns move as one element where they are adjacent and the
        // data is aligned for it.
        A.pairs = !ROWS && L.itot % 2 == 0 && reinterpret_cast<size_t>(data) % sizeof(T2) == 0;
        const int per = 2 << A.lp;
        const long long nblk = (L.nseq + per - 1)/per;
        set_smem_limit<B, body, FG_NT, 4>(FG_SMEM);
        launch_body<B, body, FG_NT, 4>(dim3((unsigned)nblk), dim3(FG_NT), bytes(A.lp), s, A);
    }

    template<typename TF>
    static void launch_fft(const FftPlan& pl, TF* data, SeqLayout L, bool inverse, TF scale, const FftFuse<TF>& fz,
                           cudaStream_t s)
    {
        const int n = pl.n;
        if (n == 1) return;
        count_launch();
        if (inverse ? launch_fixed_any<TF, true>(pl, data, L, scale, fz, s) : launch_fixed_any<TF, false>(pl, data, L, scale, fz, s))
            return;
        if (!L.rows)
        {
            if (inverse) launch_generic<TF, true, 0, false>(pl, data, L, scale, fz, s);
            else launch_generic<TF, false, 0, false>(pl, data, L, scale, fz, s);
        }
        else if (inverse)
        {
            if (fz.mode == 2) launch_generic<TF, true, 2, true>(pl, data, L, scale, fz, s);
            else launch_generic<TF, true, 0, true>(pl, data, L, scale, fz, s);
        }
        else
        {
            if (fz.mode == 1) launch_generic<TF, false, 1, true>(pl, data, L, scale, fz, s);
            else launch_generic<TF, false, 0, true>(pl, data, L, scale, fz, s);
        }
    }

    template<typename TF>
    void launch_fft_x(const FftPlan& pl, TF* data, int nrows, bool inverse, double scale, cudaStream_t s,
                      const FftFuse<TF>* fuse)
    {
        SeqLayout L; L.rows = 1; L.itot = 0; L.nseq = nrows;
        FftFuse<TF> fz;
        std::memset(&fz, 0, sizeof(fz));
        if (fuse) fz = *fuse;
        launch_fft<TF>(pl, data, L, inverse, TF(scale), fz, s);
    }

    template<typename TF>
    void launch_fft_y(const FftPlan& pl, TF* data, int itot, int jtot, int ktot, bool inverse, double scale, cudaStream_t s)
    {
        SeqLayout L; L.rows = 0; L.itot = itot; L.nseq = (long long)itot*ktot;
        FftFuse<TF> fz;
        std::memset(&fz, 0, sizeof(fz));
        launch_fft<TF>(pl, data, L, inverse, TF(scale), fz, s);
        (void)jtot;
    }

#if MHH_PREC == 64
    int fft_plan_init(FftPlan* pl, int n, cudaStream_t s)
    {
        std::memset(pl, 0, sizeof(*pl));
        pl->n = n;
        int r = n;
        for (int f : {2, 3, 5, 7}) while (r % f == 0) r /= f;
        if (r != 1) return MHH_ERR_UNSUPPORTED;
        pl->ngfac = plan_radices(n, pl->gfac);
        pl->nffac = plan_floats(n, pl->ffac);
        std::vector<double> td(2*(size_t)n);
        std::vector<float> tf(2*(size_t)n);
        const long double twopi = 6.283185307179586476925286766559005768L;
        for (int k=0; k<n; ++k)
        {
            const long double ang = -twopi*(long double)k/(long double)n;
            td[2*k] = (double)cosl(ang); td[2*k+1] = (double)sinl(ang);
            tf[2*k] = (float)td[2*k]; tf[2*k+1] = (float)td[2*k+1];
        }
        if (cudaMallocAsync((void**)&pl->tw_d, sizeof(double)*2*n, s) != cudaSuccess) return MHH_ERR_CUDA;
        if (cudaMallocAsync((void**)&pl->tw_f, sizeof(float)*2*n, s) != cudaSuccess) return MHH_ERR_CUDA;
        cudaMemcpyAsync(pl->tw_d, td.data(), sizeof(double)*2*n, cudaMemcpyHostToDevice, s);
        cudaMemcpyAsync(pl->tw_f, tf.data(), sizeof(float)*2*n, cudaMemcpyHostToDevice, s);
        return cudaStreamSynchronize(s) == cudaSuccess ? MHH_OK : MHH_ERR_CUDA;
    }

    void fft_plan_free(FftPlan* pl, cudaStream_t s)
    {
        if (pl->tw_d) cudaFreeAsync(pl->tw_d, s);
        if (pl->tw_f) cudaFreeAsync(pl->tw_f, s);
        pl->tw_d = nullptr; pl->tw_f = nullptr;
    }
#endif

    // ---------------------------------------------------------------------
    // Right-hand side, src/pres_2.cxx:155-196: divergence of ut + u/dt into
    // the packed itot*jtot*ktot array (the periodic fill of ut and vt is done
    // by the caller before).
    // ---------------------------------------------------------------------
    template<typename TF>
    __global__ void k_pres_in(Dims d, Prof<TF> pr, const TF* __restrict__ u, const TF* __restrict__ v, const TF* __restrict__ w,
                              const TF* __restrict__ ut, const TF* __restrict__ vt, const TF* __restrict__ wt,
                              TF* __restrict__ pk, TF dti)
    {
        const int i = blockIdx.x*blockDim.x + threadIdx.x;
        const int j = blockIdx.y*blockDim.y + threadIdx.y;
        const int k = blockIdx.z;
        if (i >= d.itot || j >= d.jtot) return;
        pk[i + (long long)j*d.itot + (long long)k*d.itot*d.jtot] = pres_rhs(d, pr, u, v, w, ut, vt, wt, i, j, k, dti);
    }

    template<typename TF>
    void launch_pres_in(const Dims& d, const Prof<TF>& pr, const TF* u, const TF* v, const TF* w,
                        const TF* ut, const TF* vt, const TF* wt, TF* pk, double dti, cudaStream_t s)
    {
        dim3 block(32, 8);
        dim3 grid((d.itot + 31)/32, (d.jtot + 7)/8, d.ktot);
        k_pres_in<TF><<<grid, block, 0, s>>>(d, pr, u, v, w, ut, vt, wt, pk, TF(dti));
        count_launch();
    }

    // ---------------------------------------------------------------------
    // Packed solution back into the ghost layout with the bottom ghost level
    // p[kstart-1] = p[kstart], src/pres_2.cxx:330-358 (the periodic fill
    // follows separately).
    template<typename TF>
    __global__ void k_pres_scatter(Dims d, const TF* __restrict__ pk, const TF* __restrict__ dcm, TF* __restrict__ p)
    {
        const int i = blockIdx.x*blockDim.x + threadIdx.x;
        const int j = blockIdx.y*blockDim.y + threadIdx.y;
        const int k = blockIdx.z;
        if (i >= d.itot || j >= d.jtot) return;
        const TF val = add_rn(pk[i + (long long)j*d.itot + (long long)k*d.itot*d.jtot], dcm[k]);
        const long long c = ijk(d, i + d.igc, j + d.jgc, k + d.kgc);
        p[c] = val;
        if (k == 0) p[c - d.ijcells] = val;
    }

    template<typename TF>
    void launch_pres_scatter(const Dims& d, const TF* pk, const TF* dcm, TF* p, cudaStream_t s)
    {
        dim3 block(32, 8);
        dim3 grid((d.itot + 31)/32, (d.jtot + 7)/8, d.ktot);
        k_pres_scatter<TF><<<grid, block, 0, s>>>(d, pk, dcm, p);
        count_launch();
    }

#define MHH_PRES_INST(TF) \
    template void launch_pres_in<TF>(const Dims&, const Prof<TF>&, const TF*, const TF*, const TF*, const TF*, const TF*, const TF*, TF*, double, cudaStream_t); \
    template void launch_fft_x<TF>(const FftPlan&, TF*, int, bool, double, cudaStream_t, const FftFuse<TF>*); \
    template void launch_fft_y<TF>(const FftPlan&, TF*, int, int, int, bool, double, cudaStream_t); \
    template void launch_pres_scatter<TF>(const Dims&, const TF*, const TF*, TF*, cudaStream_t);

    // Compiled once per precision (MHH_PREC, set by the build) to keep the
    // build short.
#if MHH_PREC == 64
    MHH_PRES_INST(double)
#else
    MHH_PRES_INST(float)
#endif
}
