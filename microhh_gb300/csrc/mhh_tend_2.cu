// mhh_tend_2.cu -- the DNS tendency kernel in flux form: Advec_2 + Diff_2
// (+ dry buoyancy and the large-scale pressure force), src/advec_2.cxx:80-202
// and src/diff_2.cxx:38-86.
//
// Every face flux (diffusive minus advective) is computed once.  A block owns a
// 32 x 8 tile of columns and marches upward through a chunk of levels; its 33 x
// 9 face threads compute the fluxes through the x- and y-faces of the level
// into shared memory, the 32 x 8 cell threads add the differences, and the
// vertical fluxes of the own column stay in registers.  Iteration m handles u,
// v, s at full level m and w at half level m+1.  The planes of u, v, w and s
// (1-cell halo) are staged by cp.async two levels ahead.
//
// The per-cell kernel it replaces evaluates every flux from both of its sides
// and divides by the density (1 in the Boussinesq base state, the only one):
// some 190 FP64 operations per cell against 70 here, which is what bounds the
// double form (two FP64 lanes per cycle and SM); the float form is bound by
// instruction issue.  256 x 192 x 128 per step: FP64 5.83 -> 3.01 ms, FP32 0.513
// -> 0.28 (3.44 and 0.318 before the level chunks were chosen by the busiest SM).
#include "mhh_kernels.cuh"
#include "mhh_flux.cuh"
#include "mhh_batchable.cuh"

namespace mhh
{
    namespace
    {
        constexpr int DTX = 32, DTY = 8;
        constexpr int DPW = DTX + 2, DPH = DTY + 2;
        constexpr int DPS = DPW*DPH;
        constexpr int DNX = DTX + 1, DNY = DTY + 1;
        constexpr int DNT = 320;
        constexpr int DKCHUNK_MAX = 64;
        constexpr int DNGX = DTY*DNX, DNGY = DNY*DTX;
        // Plane slots; level l of a field in slot base + l % 4.
        constexpr int DSU = 0, DSV = 4, DSW = 8, DSS = 12;
        constexpr int DPLEV = DKCHUNK_MAX + 2;

        template<typename TF, bool SCAL>
        constexpr size_t tend2_smem()
        { return sizeof(TF)*(size_t(SCAL ? 16 : 12)*DPS + 2*(SCAL ? 4 : 3)*(DNGX + DNGY) + 4*DPLEV); }
    }

    template<typename TF> struct Tend2P { Dims d; Prof<TF> pr; TendArgs<TF> a; int kchunk; };

    template<typename TF, bool SCAL, bool BUOY>
    __device__ __forceinline__ void tend2_body(const Tend2P<TF>& P, const VBlock& vb)
    {
        constexpr int NF = SCAL ? 4 : 3;
        const Dims& d = P.d;
        const Prof<TF>& pr = P.pr;
        const TendArgs<TF>& a = P.a;
        extern __shared__ __align__(16) unsigned char smem_raw[];
        TF* sm = reinterpret_cast<TF*>(smem_raw);
        TF* gxb = sm + (SCAL ? 16 : 12)*DPS;     // [2 buffers][NF][DNGX]
        TF* gyb = gxb + 2*NF*DNGX;               // [2][NF][DNGY]
        TF* lev = gyb + 2*NF*DNGY;               // [4][DPLEV]: dzhi, dzi, g/threfh, thbh

        // Warps 0-8 own the face rows fy = 0..8; warp 9 the last face column.
        const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
        const int fx = warp < DNY ? lane : DTX;
        const int fy = warp < DNY ? warp : lane;
        const bool face = warp < DNY || lane < DTY;
        const bool face_x = face && fy < DTY;
        const bool face_y = face && fx < DTX;
        const int i0 = d.istart + vb.x*DTX, j0 = d.jstart + vb.y*DTY;
        const int i = i0 + fx, j = j0 + fy;
        const bool cell = fx < DTX && fy < DTY && i < d.iend && j < d.jend;
        const int k0 = d.kstart + vb.z*P.kchunk;
        const int k1 = min(k0 + P.kchunk, d.kend);
        const int pc = (min(fy, DTY) + 1)*DPW + fx + 1;
        const int gxi = fy*DNX + fx, gyi = fy*DTX + fx;

        // 32-bit unsigned indexes, and what the fields of a level share computed
        // once (see tend_flux_body).  The (at most) two plane elements this
        // thread copies per plane; beyond the last ghost cell the last one is
        // copied, which no stored cell uses.
        const unsigned ij = (unsigned)d.ijcells;
        const int top = d.kcells - 1, e1 = tid + DNT;
        const bool two = e1 < DPS;
        unsigned go0, go1;
        {
            const int pj = tid / DPW, pi = tid - pj*DPW;
            go0 = min(i0 - 1 + pi, d.icells - 1) + (unsigned)min(j0 - 1 + pj, d.jcells - 1)*d.icells;
        }
        {
            const int pj = e1 / DPW, pi = e1 - pj*DPW;
            go1 = two ? min(i0 - 1 + pi, d.icells - 1) + (unsigned)min(j0 - 1 + pj, d.jcells - 1)*d.icells : 0u;
        }
        auto planes = [&](int l)
        {
            const unsigned lo = (unsigned)min(l, top)*ij;
            TF* dst = sm + (l & 3)*DPS + tid;
            cp_async_one(dst + DSU*DPS, a.u + (go0 + lo));
            cp_async_one(dst + DSV*DPS, a.v + (go0 + lo));
            cp_async_one(dst + DSW*DPS, a.w + (go0 + lo));
            if (SCAL) cp_async_one(dst + DSS*DPS, a.s + (go0 + lo));
            if (two)
            {
                cp_async_one(dst + DSU*DPS + DNT, a.u + (go1 + lo));
                cp_async_one(dst + DSV*DPS + DNT, a.v + (go1 + lo));
                cp_async_one(dst + DSW*DPS + DNT, a.w + (go1 + lo));
                if (SCAL) cp_async_one(dst + DSS*DPS + DNT, a.s + (go1 + lo));
            }
        };

        const int m0 = k0 - 1;
        for (int q = tid; q < P.kchunk + 2; q += DNT)
        {
            const int l = min(m0 + q, top);
            lev[0*DPLEV + q] = pr.dzhi[l];
            lev[1*DPLEV + q] = pr.dzi[l];
            if (BUOY) { lev[2*DPLEV + q] = TF(GRAV)/pr.threfh[l]; lev[3*DPLEV + q] = pr.thbh[l]; }
        }
        for (int l = m0; l <= m0 + 2; ++l) planes(l);
        cp_async_commit();

        const unsigned col = cell ? (unsigned)(i + j*d.icells) : 0u;
        const TF visc = a.visc, svisc = a.svisc;
        const TF dxi = dxi_of<TF>(d), dyi = dyi_of<TF>(d);
        // Factors of the differences and of the products of sums.
        const TF vx = visc*dxi, vy = visc*dyi, sx = svisc*dxi, sy = svisc*dyi;
        const TF q4 = TF(-0.25), q2 = TF(-0.5);
        TF zu_b = 0, zv_b = 0, zw_b = 0, zs_b = 0;

        cp_async_wait_all();
        __syncthreads();

        for (int m = m0; m < k1; ++m)
        {
            const int buf = (m - m0) & 1, lq = m - m0;
            TF* gx = gxb + buf*NF*DNGX;
            TF* gy = gyb + buf*NF*DNGY;
            const TF* L0 = sm + (m & 3)*DPS + pc;
            const TF* L1 = sm + ((m + 1) & 3)*DPS + pc;
            const TF* U0 = L0 + DSU*DPS; const TF* U1 = L1 + DSU*DPS;
            const TF* V0 = L0 + DSV*DPS; const TF* V1 = L1 + DSV*DPS;
            const TF* W1 = L1 + DSW*DPS;
            const TF* S0 = L0 + DSS*DPS; const TF* S1 = L1 + DSS*DPS;
            // The planes of level m+3, first used two iterations on, into the
            // slots that iteration m-1 freed.
            if (m + 2 < k1) planes(m + 3);
            cp_async_commit();

            const bool wlev = m+1 > d.kstart && m+1 < d.kend;
            const bool write = cell && m >= k0;
            const unsigned c = col + (unsigned)m*ij;
            TF tu = 0, tv = 0, tw = 0, ts = 0, w2 = 0;
            if (write)
            {
                tu = a.ut[c]; tv = a.vt[c];
                if (wlev) tw = a.wt[c + ij];
                if (SCAL) ts = a.st[c];
            }
            if (cell && m + 2 < d.kcells) w2 = __ldg(a.w + (c + 2u*ij));

            if (face)
            {
                const TF u0 = U0[0], v0 = V0[0], w1 = W1[0], u1 = U1[0], v1 = V1[0];
                const TF uw = U0[-1], us = U0[-DPW], vw = V0[-1], vs = V0[-DPW];
                if (face_x)
                {
                    const TF s = uw + u0, ww = W1[-1];
                    gx[0*DNGX + gxi] = fma(s*s, q4, (u0 - uw)*(vx));
                    gx[1*DNGX + gxi] = fma((us + u0)*(vw + v0), q4, (v0 - vw)*vx);
                    gx[2*DNGX + gxi] = fma((u0 + u1)*(ww + w1), q4, (w1 - ww)*vx);
                    if (SCAL)
                    {
                        const TF sw = S0[-1], s0 = S0[0];
                        gx[3*DNGX + gxi] = fma(u0*(sw + s0), q2, (s0 - sw)*sx);
                    }
                }
                if (face_y)
                {
                    const TF s = vs + v0, ws = W1[-DPW];
                    gy[0*DNGY + gyi] = fma((vw + v0)*(us + u0), q4, (u0 - us)*vy);
                    gy[1*DNGY + gyi] = fma(s*s, q4, (v0 - vs)*vy);
                    gy[2*DNGY + gyi] = fma((v0 + v1)*(ws + w1), q4, (w1 - ws)*vy);
                    if (SCAL)
                    {
                        const TF ss = S0[-DPW], s0 = S0[0];
                        gy[3*DNGY + gyi] = fma(v0*(ss + s0), q2, (s0 - ss)*sy);
                    }
                }
            }
            // Vertical faces of the own column: half level m+1 for u, v, s, full
            // level m+1 for w.
            TF zu_t = 0, zv_t = 0, zw_t = 0, zs_t = 0, buoy = 0;
            if (cell)
            {
                const TF dzh = lev[0*DPLEV + lq + 1], dz = lev[1*DPLEV + lq + 1];
                const TF u0 = U0[0], u1 = U1[0], v0 = V0[0], v1 = V1[0], w1 = W1[0];
                const TF vz = visc*dzh;
                zu_t = fma((W1[-1] + w1)*(u0 + u1), q4, (u1 - u0)*vz);
                zv_t = fma((W1[-DPW] + w1)*(v0 + v1), q4, (v1 - v0)*vz);
                const TF s = w1 + w2;
                zw_t = fma(s*s, q4, (w2 - w1)*(visc*dz));
                if (SCAL) zs_t = fma(w1*(S0[0] + S1[0]), q2, (S1[0] - S0[0])*(svisc*dzh));
                if (BUOY && wlev)
                {
                    const TF sb = SCAL ? S0[0] : __ldg(a.s + c), st = SCAL ? S1[0] : __ldg(a.s + (c + ij));
                    buoy = lev[2*DPLEV + lq + 1]*(i2(sb, st) - lev[3*DPLEV + lq + 1]);
                }
            }

            // The planes of iteration m+1 were issued two iterations ago.
            asm volatile("cp.async.wait_group 1;\n" ::: "memory");
            __syncthreads();

            if (write)
            {
                const TF dz = lev[1*DPLEV + lq], dzh = lev[0*DPLEV + lq + 1];
                auto total = [&](int f, TF t, TF zb, TF zt, TF zi)
                {
                    const TF* x = gx + f*DNGX + gxi;
                    const TF* y = gy + f*DNGY + gyi;
                    return fma(zt - zb, zi, fma(y[DTX] - y[0], dyi, fma(x[1] - x[0], dxi, t)));
                };
                a.ut[c] = total(0, tu + a.fbody, zu_b, zu_t, dz);
                a.vt[c] = total(1, tv, zv_b, zv_t, dz);
                if (wlev) a.wt[c + ij] = total(2, tw + buoy, zw_b, zw_t, dzh);
                if (SCAL) a.st[c] = total(3, ts, zs_b, zs_t, dz);
            }
            zu_b = zu_t; zv_b = zv_t; zw_b = zw_t; zs_b = zs_t;
        }
        cp_async_wait_all();
    }

    template<typename TF, bool SCAL, bool BUOY>
    static void launch_t2(const Dims& d, const Prof<TF>& pr, const TendArgs<TF>& a, int kchunk, cudaStream_t s)
    {
        constexpr size_t smem = tend2_smem<TF, SCAL>();
        const int nx = (d.itot + DTX - 1)/DTX, ny = (d.jtot + DTY - 1)/DTY;
        constexpr int occ = sizeof(TF) == 4 ? 3 : 2;
        kchunk = auto_kchunk(kchunk, (long long)nx*ny, d.ktot, sizeof(TF) == 8, DKCHUNK_MAX);
        launch_body<Tend2P<TF>, tend2_body<TF, SCAL, BUOY>, DNT, occ>(
            dim3(nx, ny, (d.ktot + kchunk - 1)/kchunk), dim3(DNT), smem, s, Tend2P<TF>{d, pr, a, kchunk});
        count_launch();
    }

    template<typename TF>
    void launch_tendency_2(const Dims& d, const Prof<TF>& pr, const TendArgs<TF>& a, bool scal, bool buoy, bool force,
                           int kchunk, cudaStream_t s)
    {
        TendArgs<TF> b = a;
        if (!force) b.fbody = TF(0);
        if (scal && buoy) launch_t2<TF, true, true>(d, pr, b, kchunk, s);
        else if (scal) launch_t2<TF, true, false>(d, pr, b, kchunk, s);
        else if (buoy) launch_t2<TF, false, true>(d, pr, b, kchunk, s);
        else launch_t2<TF, false, false>(d, pr, b, kchunk, s);
    }

    template void launch_tendency_2<double>(const Dims&, const Prof<double>&, const TendArgs<double>&, bool, bool, bool, int, cudaStream_t);
    template void launch_tendency_2<float>(const Dims&, const Prof<float>&, const TendArgs<float>&, bool, bool, bool, int, cudaStream_t);
}
