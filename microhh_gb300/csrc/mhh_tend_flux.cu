// mhh_tend_flux.cu -- the LES tendency kernel in flux form (Advec_2i5 +
// Smagorinsky diffusion + dry buoyancy, optionally with the Monin-Obukhov
// wall fluxes).
//
// Every face flux is computed once.  A block owns a 32 x 8 tile of columns
// and marches upward through a chunk of levels.  Its 33 x 9 face threads
// compute, per level, the total (diffusive minus advective) flux through the
// x- and y-faces of the u, v, w and s control volumes into shared memory; the
// 32 x 8 cell threads add the flux differences, with the vertical faces of
// their own column kept in registers (the top face of one level is the bottom
// face of the next).  The shear stresses are shared between the fields whose
// faces coincide: tau_xy at (i-1/2, j-1/2) is the y-flux of u and the x-flux
// of v, tau_xz at (i-1/2, k+1/2) the x-flux of w and the z-flux of u, and
// tau_yz likewise for w and v.
//
// Iteration m handles u, v, s at full level m and w at half level m+1, so the
// horizontal faces of w and the vertical faces of u, v, s lie on the same
// half level and share tau_xz and tau_yz.  The planes of each level (u, v, w,
// s and the eddy viscosity with a 3-cell halo) are staged in shared memory
// by cp.async two levels ahead of their use; the 7-point vertical
// neighbourhoods of the own column come from register queues.
//
// The arithmetic per face is that of the reference's kernels:
// src/advec_2i5.cxx:150-728 (6th-order interpolation with 5th-order upwind
// dissipation, lower orders next to the walls), include/diff_kernels.h:144-484
// (Smagorinsky fluxes; wall fluxes from the surface model) and
// src/thermo_dry.cxx:165-181 (buoyancy); with LIM the scalar's advective
// fluxes are those of the flux limiter (include/advec_monotonic.h:28-219).
// The sum of all fluxes is formed
// before it is added to the tendency, so the result differs from the
// reference's term-by-term accumulation by round-off only.
#include "mhh_kernels.cuh"
#include "mhh_stencil.cuh"
#include "mhh_flux.cuh"
#include "mhh_batchable.cuh"

namespace mhh
{
    namespace
    {
        constexpr int FTX = 32, FTY = 8, FH = 3;
        constexpr int FPW = 40;                 // plane row (FTX + 2*FH, padded)
        constexpr int FPH = FTY + 2*FH;         // plane rows
        constexpr int FPS = FPW*FPH;            // plane size
        constexpr int NFX = FTX + 1, NFY = FTY + 1;
        constexpr int NTHR = 320;
        constexpr int FKCHUNK_MAX = 64;
        // Plane slots: four per field; level l of a field lives in slot
        // base + l % 4, so that the planes of one level sit at one offset from
        // their fields' bases.  Planes are prefetched two levels ahead.
        constexpr int SU = 0, SV = 4, SW = 8, SS = 12, SE = 16, NSLOT = 20;
        constexpr int NGX = FTY*NFX;            // x-faces per level and field
        constexpr int NGY = NFY*FTX;            // y-faces per level and field
        constexpr int NEL1 = FPS - NTHR;        // threads that copy a second element

        template<typename TF> struct FluxOcc { static constexpr int v = sizeof(TF) == 4 ? 2 : 1; };

        constexpr int NPROF = 8;                // per-level constants staged in shared memory
        constexpr int PLEV = FKCHUNK_MAX + 2;   // levels m0 .. m0+kchunk+1

        template<typename TF>
        size_t flux_smem() { return sizeof(TF)*(size_t(NSLOT)*FPS + 2*4*(NGX + NGY) + NPROF*PLEV); }
    }

    template<typename TF> struct TendFluxP { Dims d; Prof<TF> pr; TendArgs<TF> a; int kchunk; };

    // ADV, DIF: with one of them false the other term alone (the module calls of
    // Advec_2i5 and Diff_smag2; the per-cell kernels they replace evaluate every
    // flux from both sides.  Step by modules, ms: float 96 x 96 x 64 0.686, now
    // 0.663, 256 x 256 x 128 4.66, now 3.33; FP64 3.52, now 2.05 and 42.1, now
    // 21.5).
    template<typename TF, bool SURF, bool SCAL, bool BUOY, bool LIM, bool ADV = true, bool DIF = true>
    __device__ __forceinline__ void tend_flux_body(const TendFluxP<TF>& P, const VBlock& vb)
    {
        const Dims& d = P.d;
        const Prof<TF>& pr = P.pr;
        const TendArgs<TF>& a = P.a;
        const int kchunk = P.kchunk;
        extern __shared__ __align__(16) unsigned char smem_raw[];
        TF* sm = reinterpret_cast<TF*>(smem_raw);
        TF* gbase = sm + NSLOT*FPS;     // [2 buffers][NGX][4 fields] then [2][NGY][4]
        TF* prof = gbase + 2*4*(NGX + NGY);   // [NPROF][PLEV]

        // Warps 0-8 own the face rows fy = 0..8 (fx = lane); warp 9 owns the
        // last face column fx = 32 of the rows fy = 0..7.  A warp thus reads
        // one contiguous plane row.
        const int tid = threadIdx.x;
        const int warp = tid >> 5, lane = tid & 31;
        const int fx = warp < NFY ? lane : FTX;
        const int fy = warp < NFY ? warp : lane;
        const bool face = warp < NFY || lane < FTY;
        const bool face_x = face && fy < FTY;
        const bool face_y = face && fx < FTX;
        const int i0 = d.istart + vb.x*FTX;
        const int j0 = d.jstart + vb.y*FTY;
        const int i = i0 + fx, j = j0 + fy;
        const bool cell = fx < FTX && fy < FTY && i < d.iend && j < d.jend;
        const int k0 = d.kstart + vb.z*kchunk;
        const int k1 = min(k0 + kchunk, d.kend);
        const int pc = (min(fy, FTY) + FH)*FPW + (fx + FH);   // own (i, j) in a plane
        const int gxi = fy*NFX + fx, gyi = fy*FTX + fx;

        // Indexes into the fields are 32-bit and unsigned (fewer than 2^32 cells),
        // and whatever the fields of a level share is computed once: with 64-bit
        // offsets per field, slots modulo 3 and bounds tests per copy, integer
        // and uniform instructions were nearly half of the 761 a cell took in
        // float (now 630; 5.16 -> 4.81 ms per step at 512 x 512 x 256).
        //
        // The (at most) two plane elements this thread copies per plane.  Beyond
        // the last ghost cell the last one is copied; no stored cell uses it.
        const unsigned ij = (unsigned)d.ijcells;
        const int top = d.kcells - 1;
        const int e1 = tid + NTHR;
        const bool two = tid < NEL1;
        unsigned go0, go1;
        {
            const int pj = tid / FPW, pi = tid - pj*FPW;
            go0 = min(i0 - FH + pi, d.icells - 1) + (unsigned)min(j0 - FH + pj, d.jcells - 1)*d.icells;
        }
        {
            const int pj = e1 / FPW, pi = e1 - pj*FPW;
            go1 = two ? min(i0 - FH + pi, d.icells - 1) + (unsigned)min(j0 - FH + pj, d.jcells - 1)*d.icells : 0u;
        }
        // Plane of field f (level offset lo, slot offset so) into the slots from
        // base on.
        auto plane = [&](int base, const TF* f, unsigned lo, int so)
        {
            TF* dst = sm + base*FPS + so + tid;
            cp_async_one(dst, f + (go0 + lo));
            if (two) cp_async_one(dst + NTHR, f + (go1 + lo));
        };

        const TF* __restrict__ u = a.u;
        const TF* __restrict__ v = a.v;
        const TF* __restrict__ w = a.w;
        const TF* __restrict__ s = a.s;
        const TF* __restrict__ ev = a.evisc;
        const unsigned col = cell ? (unsigned)(i + j*d.icells) : 0u;
        // Offset of level l, clamped to the levels there are.
        auto level = [&](int l) { return (unsigned)min(max(l, 0), top)*ij; };

        // Per-level constants of the chunk: index l - m0 for level l.
        const int m0 = k0 - 1;
        for (int q = tid; q < kchunk + 2; q += NTHR)
        {
            const int l = min(m0 + q, top);
            prof[0*PLEV + q] = pr.dzhi[l];
            prof[1*PLEV + q] = pr.rhorefh[l];
            prof[2*PLEV + q] = pr.rhoref[l];
            prof[3*PLEV + q] = pr.dzi[l];
            prof[4*PLEV + q] = TF(GRAV)/pr.threfh[l];
            prof[7*PLEV + q] = pr.thbh[l];
            prof[5*PLEV + q] = pr.zfac[l];
            prof[6*PLEV + q] = pr.zfach[l];
        }

        // Planes of the first three iterations (m0 .. m0+2).
        for (int l = m0; l <= m0+3; ++l)
        {
            const unsigned lo = level(l);
            const int so = (l & 3)*FPS;
            plane(SU, u, lo, so); plane(SV, v, lo, so); plane(SW, w, lo, so);
            if (DIF) plane(SE, ev, lo, so);
            if (SCAL && l < m0+3) plane(SS, s, lo, so);
        }
        cp_async_commit();

        // Register queues of the own column: u, v, s hold levels m-2 .. m+3,
        // w holds m-1 .. m+4.
        TF qu[6], qv[6], qw[6], qs[6];
        if (cell)
        {
            #pragma unroll
            for (int q=0; q<6; ++q)
            {
                const unsigned l = col + level(m0 - 2 + q);
                qu[q] = __ldg(u + l);
                qv[q] = __ldg(v + l);
                qw[q] = __ldg(w + (col + level(m0 - 1 + q)));
                qs[q] = (SCAL || BUOY) ? __ldg(s + l) : TF(0);
            }
        }
        TF ufb = 0, uft = 0, vfb = 0, vft = 0, sfb = 0, sft = 0;
        if (SURF && cell)
        {
            ufb = a.u_fluxbot[col]; uft = a.u_fluxtop[col];
            vfb = a.v_fluxbot[col]; vft = a.v_fluxtop[col];
            if (SCAL) { sfb = a.s_fluxbot[col]; sft = a.s_fluxtop[col]; }
        }

        const TF dxi = dxi_of<TF>(d), dyi = dyi_of<TF>(d);
        const TF visc = a.visc, svisc = a.svisc, tpri = a.tpri;
        TF gzu_b = 0, gzv_b = 0, gzw_b = 0, gzs_b = 0;

        cp_async_wait_all();
        __syncthreads();

        // Double form: the viscosity sums of the own faces at levels m and m+1.
        TF ex0 = 0, ey0 = 0, ex1 = 0, ey1 = 0;
        if (sizeof(TF) == 8 && DIF && face)
        {
            const TF* E = sm + SE*FPS + (m0 & 3)*FPS + pc;
            ex0 = E[-1] + E[0];
            ey0 = E[-FPW] + E[0];
        }

        for (int m = m0; m < k1; ++m)
        {
            const int buf = (m - m0) & 1;
            TF* gx = gbase + buf*4*NGX;
            TF* gy = gbase + 2*4*NGX + buf*4*NGY;
            // Own point in the planes of levels m and m+1.
            const TF* L0 = sm + (m & 3)*FPS + pc;
            const TF* L1 = sm + ((m + 1) & 3)*FPS + pc;
            const TF* U0 = L0 + SU*FPS; const TF* U1 = L1 + SU*FPS;
            const TF* V0 = L0 + SV*FPS; const TF* V1 = L1 + SV*FPS;
            const TF* W1 = L1 + SW*FPS;
            const TF* S0 = L0 + SS*FPS;
            const TF* E0 = L0 + SE*FPS; const TF* E1 = L1 + SE*FPS;
            #define PL(P, dx, dy) (P)[(dy)*FPW + (dx)]

            const bool write = cell && m >= k0;
            const bool wlev = m+1 > d.kstart && m+1 < d.kend;
            const unsigned c = col + (unsigned)m*ij;
            // Early loads: the tendencies this iteration updates and the queue
            // entries of the next iteration.
            TF tu = 0, tv = 0, tw = 0, ts = 0;
            if (write)
            {
                tu = a.ut[c]; tv = a.vt[c];
                if (wlev) tw = a.wt[c + ij];
                if (SCAL) ts = a.st[c];
            }
            const unsigned lo4 = (unsigned)min(m + 4, top)*ij;
            TF nu = 0, nv = 0, nw = 0, ns = 0;
            if (cell)
            {
                nu = __ldg(u + (col + lo4)); nv = __ldg(v + (col + lo4));
                nw = __ldg(w + (col + (unsigned)min(m + 5, top)*ij));
                if (SCAL || BUOY) ns = __ldg(s + (col + lo4));
            }

            const TF* pl = prof + (m + 1 - m0);      // constants of level m+1
            const TF dzhi1 = pl[0*PLEV];

            // ---- faces: shear stresses and total fluxes ----
            TF txz = 0, tyz = 0;
            if (face)
            {
                if constexpr (sizeof(TF) == 4)
                {
                    const float2 zero = make_float2(0.f, 0.f);
                    const TF txy = !DIF ? TF(0) : (TF(0.25)*(PL(E0,-1,-1) + PL(E0,0,-1) + PL(E0,-1,0) + PL(E0,0,0)) + visc)
                                 * ((PL(U0,0,0) - PL(U0,0,-1))*dyi + (PL(V0,0,0) - PL(V0,-1,0))*dxi);
                    // tau_xz and tau_yz in one packed pair.
                    const float2 ez = __ffma2_rn(__fadd2_rn(__fadd2_rn(f2(PL(E0,-1,0), PL(E0,0,-1)), f2(PL(E0,0,0), PL(E0,0,0))),
                                                            __fadd2_rn(f2(PL(E1,-1,0), PL(E1,0,-1)), f2(PL(E1,0,0), PL(E1,0,0)))),
                                                 f2(0.25f, 0.25f), f2(visc, visc));
                    const float2 gz = __ffma2_rn(sub2(f2(PL(U1,0,0), PL(V1,0,0)), f2(PL(U0,0,0), PL(V0,0,0))), f2(dzhi1, dzhi1),
                                                 __fmul2_rn(sub2(f2(PL(W1,0,0), PL(W1,0,0)), f2(PL(W1,-1,0), PL(W1,0,-1))),
                                                            f2(dxi, dyi)));
                    const float2 tz = DIF ? __fmul2_rn(ez, gz) : zero;
                    txz = tz.x; tyz = tz.y;
                    // Float form: the x- and y-face advective fluxes of each
                    // field in packed pairs (both computed by every face
                    // thread; the plane holds the stencils of the edge faces).
                    const float2 Au = !ADV ? zero : adv6x2(make_float2(i2(PL(U0,-1,0), PL(U0,0,0)), i2(PL(V0,-1,0), PL(V0,0,0))),
                                             make_float2(PL(U0,-3,0), PL(U0,0,-3)), make_float2(PL(U0,-2,0), PL(U0,0,-2)),
                                             make_float2(PL(U0,-1,0), PL(U0,0,-1)), make_float2(PL(U0,0,0), PL(U0,0,0)),
                                             make_float2(PL(U0,1,0), PL(U0,0,1)), make_float2(PL(U0,2,0), PL(U0,0,2)));
                    const float2 Av = !ADV ? zero : adv6x2(make_float2(i2(PL(U0,0,-1), PL(U0,0,0)), i2(PL(V0,0,-1), PL(V0,0,0))),
                                             make_float2(PL(V0,-3,0), PL(V0,0,-3)), make_float2(PL(V0,-2,0), PL(V0,0,-2)),
                                             make_float2(PL(V0,-1,0), PL(V0,0,-1)), make_float2(PL(V0,0,0), PL(V0,0,0)),
                                             make_float2(PL(V0,1,0), PL(V0,0,1)), make_float2(PL(V0,2,0), PL(V0,0,2)));
                    const float2 Aw = !ADV ? zero : adv6x2(make_float2(i2(PL(U0,0,0), PL(U1,0,0)), i2(PL(V0,0,0), PL(V1,0,0))),
                                             make_float2(PL(W1,-3,0), PL(W1,0,-3)), make_float2(PL(W1,-2,0), PL(W1,0,-2)),
                                             make_float2(PL(W1,-1,0), PL(W1,0,-1)), make_float2(PL(W1,0,0), PL(W1,0,0)),
                                             make_float2(PL(W1,1,0), PL(W1,0,1)), make_float2(PL(W1,2,0), PL(W1,0,2)));
                    float2 As = zero;
                    if (SCAL && ADV)
                    {
                        if (LIM)
                            As = make_float2(lim_flux(PL(U0,0,0), PL(S0,-2,0), PL(S0,-1,0), PL(S0,0,0), PL(S0,1,0), 0),
                                             lim_flux(PL(V0,0,0), PL(S0,0,-2), PL(S0,0,-1), PL(S0,0,0), PL(S0,0,1), 0));
                        else
                            As = adv6x2(make_float2(PL(U0,0,0), PL(V0,0,0)),
                                        make_float2(PL(S0,-3,0), PL(S0,0,-3)), make_float2(PL(S0,-2,0), PL(S0,0,-2)),
                                        make_float2(PL(S0,-1,0), PL(S0,0,-1)), make_float2(PL(S0,0,0), PL(S0,0,0)),
                                        make_float2(PL(S0,1,0), PL(S0,0,1)), make_float2(PL(S0,2,0), PL(S0,0,2)));
                    }
                    // Normal diffusive fluxes of u (x) and v (y), and of s in
                    // x and y, in packed pairs.
                    const float2 eo = f2(PL(E0,-1,0), PL(E0,0,-1));
                    const float2 h2 = f2(dxi, dyi);
                    const float2 Duv = !DIF ? zero : __fmul2_rn(__fmul2_rn(__fadd2_rn(eo, f2(visc, visc)), f2(2.f, 2.f)),
                                                  __fmul2_rn(sub2(f2(PL(U0,0,0), PL(V0,0,0)), f2(PL(U0,-1,0), PL(V0,0,-1))), h2));
                    float2 Ds = zero;
                    if (SCAL && DIF)
                        Ds = __fmul2_rn(__ffma2_rn(__fmul2_rn(__fadd2_rn(eo, f2(PL(E0,0,0), PL(E0,0,0))), f2(0.5f, 0.5f)),
                                                   f2(tpri, tpri), f2(svisc, svisc)),
                                        __fmul2_rn(sub2(f2(PL(S0,0,0), PL(S0,0,0)), f2(PL(S0,-1,0), PL(S0,0,-1))), h2));
                    // The four fields' fluxes of a face are adjacent: one
                    // 16-byte store per face.
                    if (face_x)
                        reinterpret_cast<float4*>(gx)[gxi] = make_float4(Duv.x - Au.x, txy - Av.x, txz - Aw.x,
                                                                         SCAL ? Ds.x - As.x : 0.f);
                    if (face_y)
                        reinterpret_cast<float4*>(gy)[gyi] = make_float4(txy - Au.y, Duv.y - Av.y, tyz - Aw.y,
                                                                         SCAL ? Ds.y - As.y : 0.f);
                }
                else
                {
                    // Double form, bound by the FP64 pipe: sums of the eddy
                    // viscosity at the face's two cells shared between the
                    // stresses and carried up a level, constant factors
                    // folded, each flux one FMA off its advective part.
                    if (DIF) { ex1 = PL(E1,-1,0) + PL(E1,0,0); ey1 = PL(E1,0,-1) + PL(E1,0,0); }
                    const TF txy = !DIF ? TF(0) : fma(ex0 + (PL(E0,-1,-1) + PL(E0,0,-1)), TF(0.25), visc)
                                 * fma(PL(V0,0,0) - PL(V0,-1,0), dxi, (PL(U0,0,0) - PL(U0,0,-1))*dyi);
                    if (face_x)
                    {
                        if (DIF) txz = fma(ex0 + ex1, TF(0.25), visc)
                            * fma(PL(W1,0,0) - PL(W1,-1,0), dxi, (PL(U1,0,0) - PL(U0,0,0))*dzhi1);
                        // u at the cell centre i-1.
                        {
                            const TF uw = PL(U0,-1,0) + PL(U0,0,0);
                            const TF A = (!ADV ? TF(0) : uw*upwind5<true>(uw, PL(U0,-3,0), PL(U0,-2,0), PL(U0,-1,0), PL(U0,0,0), PL(U0,1,0), PL(U0,2,0)));
                            gx[(gxi)*4 + 0] = DIF ? fma(fma(PL(E0,-1,0), TF(2)*dxi, TF(2)*dxi*visc), PL(U0,0,0) - PL(U0,-1,0), -A) : -A;
                        }
                        // v at (i-1/2, j-1/2).
                        {
                            const TF uw = PL(U0,0,-1) + PL(U0,0,0);
                            gx[(gxi)*4 + 1] = ADV ? fma(-uw, upwind5<true>(uw, PL(V0,-3,0), PL(V0,-2,0), PL(V0,-1,0), PL(V0,0,0), PL(V0,1,0), PL(V0,2,0)), txy) : txy;
                        }
                        // w at (i-1/2, m+1/2).
                        {
                            const TF uw = PL(U0,0,0) + PL(U1,0,0);
                            gx[(gxi)*4 + 2] = ADV ? fma(-uw, upwind5<true>(uw, PL(W1,-3,0), PL(W1,-2,0), PL(W1,-1,0), PL(W1,0,0), PL(W1,1,0), PL(W1,2,0)), txz) : txz;
                        }
                        if (SCAL)
                        {
                            const TF uw = PL(U0,0,0);
                            const TF A = LIM && ADV ? lim_flux(uw, PL(S0,-2,0), PL(S0,-1,0), PL(S0,0,0), PL(S0,1,0), 0)
                                             : (!ADV ? TF(0) : uw*upwind5<false>(uw, PL(S0,-3,0), PL(S0,-2,0), PL(S0,-1,0), PL(S0,0,0), PL(S0,1,0), PL(S0,2,0)));
                            gx[(gxi)*4 + 3] = DIF ? fma(fma(ex0, TF(0.5)*tpri*dxi, svisc*dxi), PL(S0,0,0) - PL(S0,-1,0), -A) : -A;
                        }
                    }
                    if (face_y)
                    {
                        if (DIF) tyz = fma(ey0 + ey1, TF(0.25), visc)
                            * fma(PL(W1,0,0) - PL(W1,0,-1), dyi, (PL(V1,0,0) - PL(V0,0,0))*dzhi1);
                        // u at (i-1/2, j-1/2).
                        {
                            const TF vs = PL(V0,-1,0) + PL(V0,0,0);
                            gy[(gyi)*4 + 0] = ADV ? fma(-vs, upwind5<true>(vs, PL(U0,0,-3), PL(U0,0,-2), PL(U0,0,-1), PL(U0,0,0), PL(U0,0,1), PL(U0,0,2)), txy) : txy;
                        }
                        // v at the cell centre j-1.
                        {
                            const TF vs = PL(V0,0,-1) + PL(V0,0,0);
                            const TF A = (!ADV ? TF(0) : vs*upwind5<true>(vs, PL(V0,0,-3), PL(V0,0,-2), PL(V0,0,-1), PL(V0,0,0), PL(V0,0,1), PL(V0,0,2)));
                            gy[(gyi)*4 + 1] = DIF ? fma(fma(PL(E0,0,-1), TF(2)*dyi, TF(2)*dyi*visc), PL(V0,0,0) - PL(V0,0,-1), -A) : -A;
                        }
                        // w at (j-1/2, m+1/2).
                        {
                            const TF vs = PL(V0,0,0) + PL(V1,0,0);
                            gy[(gyi)*4 + 2] = ADV ? fma(-vs, upwind5<true>(vs, PL(W1,0,-3), PL(W1,0,-2), PL(W1,0,-1), PL(W1,0,0), PL(W1,0,1), PL(W1,0,2)), tyz) : tyz;
                        }
                        if (SCAL)
                        {
                            const TF vs = PL(V0,0,0);
                            const TF A = LIM && ADV ? lim_flux(vs, PL(S0,0,-2), PL(S0,0,-1), PL(S0,0,0), PL(S0,0,1), 0)
                                             : (!ADV ? TF(0) : vs*upwind5<false>(vs, PL(S0,0,-3), PL(S0,0,-2), PL(S0,0,-1), PL(S0,0,0), PL(S0,0,1), PL(S0,0,2)));
                            gy[(gyi)*4 + 3] = DIF ? fma(fma(ey0, TF(0.5)*tpri*dyi, svisc*dyi), PL(S0,0,0) - PL(S0,0,-1), -A) : -A;
                        }
                    }
                }
            }

            // ---- vertical faces of the own column ----
            TF gzu_t = 0, gzv_t = 0, gzw_t = 0, gzs_t = 0, buoy = 0;
            if (cell)
            {
                const int kf = m + 1;
                const int ot = ADV ? face_order_full(d, kf) : 0;      // 0: no advective flux
                const TF rhoh1 = pl[1*PLEV];
                // u and v: diffusive flux from the shear stress of the same
                // face, or the surface model's flux at the walls.
                const TF du = (SURF && kf == d.kstart) ? -ufb : ((SURF && kf == d.kend) ? -uft : txz);
                const TF dv = (SURF && kf == d.kstart) ? -vfb : ((SURF && kf == d.kend) ? -vft : tyz);
                if constexpr (sizeof(TF) == 4)
                {
                    const float2 A = zadv2(qu, qv, f2(i2(PL(W1,-1,0), PL(W1,0,0)), i2(PL(W1,0,-1), PL(W1,0,0))), ot);
                    const float2 g = __fmul2_rn(f2(rhoh1, rhoh1), sub2(f2(du, dv), A));
                    gzu_t = g.x; gzv_t = g.y;
                }
                else
                {
                    const TF wu = PL(W1,-1,0) + PL(W1,0,0), wv = PL(W1,0,-1) + PL(W1,0,0);
                    if (ot == 6)
                    {
                        gzu_t = rhoh1*fma(-wu, upwind5<true>(wu, qu[0], qu[1], qu[2], qu[3], qu[4], qu[5]), du);
                        gzv_t = rhoh1*fma(-wv, upwind5<true>(wv, qv[0], qv[1], qv[2], qv[3], qv[4], qv[5]), dv);
                    }
                    else
                    {
                        gzu_t = rhoh1*(du - zadv(qu, TF(0.5)*wu, ot));
                        gzv_t = rhoh1*(dv - zadv(qv, TF(0.5)*wv, ot));
                    }
                }
                // Float form, interior levels: the vertical advective fluxes of
                // w (through full level kf) and of s (through half level kf),
                // both 6th/5th order, in one packed pair.
                bool paired = false;
                float2 aws = make_float2(0.f, 0.f);
                if constexpr (sizeof(TF) == 4 && SCAL && !LIM)
                {
                    if (ot == 6 && kf < d.kend && face_order_w(d, kf) == 6)
                    {
                        aws = adv6x2(f2(i2(qw[2], qw[3]), qw[2]), f2(qw[0], qs[0]), f2(qw[1], qs[1]), f2(qw[2], qs[2]),
                                     f2(qw[3], qs[3]), f2(qw[4], qs[4]), f2(qw[5], qs[5]));
                        paired = true;
                    }
                }
                if (SCAL)
                {
                    const TF ds = (SURF && kf == d.kstart) ? -sfb : ((SURF && kf == d.kend) ? -sft
                                : (DIF ? (TF(0.5)*(PL(E0,0,0) + PL(E1,0,0))*tpri + svisc)*(qs[3] - qs[2])*dzhi1 : TF(0)));
                    TF as;
                    if (paired) as = aws.y;
                    else if (LIM)
                    {
                        const int side = kf == d.kstart+1 ? -1 : (kf == d.kend-1 ? 1 : 0);
                        as = ot ? lim_flux(qw[2], qs[1], qs[2], qs[3], qs[4], side) : TF(0);
                    }
                    else if (sizeof(TF) == 8 && ot == 6)
                        as = qw[2]*upwind5<false>(qw[2], qs[0], qs[1], qs[2], qs[3], qs[4], qs[5]);
                    else as = zadv(qs, qw[2], ot);
                    gzs_t = rhoh1*(ds - as);
                }
                // w: the full level kf between w(kf) and w(kf+1).
                if (kf < d.kend)
                {
                    const int ow = face_order_w(d, kf);
                    const TF dw = !DIF ? TF(0) : TF(2)*(PL(E1,0,0) + visc)*(qw[3] - qw[2])*pl[3*PLEV];
                    TF aw;
                    if (!ADV) aw = TF(0);
                    else if (paired) aw = aws.x;
                    else if (sizeof(TF) == 8 && ow == 6)
                    {
                        const TF ww = qw[2] + qw[3];
                        aw = ww*upwind5<true>(ww, qw[0], qw[1], qw[2], qw[3], qw[4], qw[5]);
                    }
                    else if (ow == 6) aw = adv6(i2(qw[2], qw[3]), qw[0], qw[1], qw[2], qw[3], qw[4], qw[5]);
                    else if (ow == 4) aw = i2(qw[2], qw[3])*i4ws(qw[1], qw[2], qw[3], qw[4])
                                         - fabs(i2(qw[2], qw[3]))*i3ws(qw[1], qw[2], qw[3], qw[4]);
                    else aw = i2(qw[2], qw[3])*i2(qw[2], qw[3]);
                    gzw_t = pl[2*PLEV]*(dw - aw);
                }
                if (BUOY && wlev)
                    buoy = pl[4*PLEV]*(i2(qs[2], qs[3]) - pl[7*PLEV]);
            }
            #undef PL

            // The planes of iteration m+1 were issued two iterations ago; the
            // last iteration's group may stay in flight.
            asm volatile("cp.async.wait_group 1;\n" ::: "memory");
            __syncthreads();

            // Planes first used by iteration m+3 into the slots that
            // iteration m freed.
            if (m + 3 < k1)
            {
                const int so = (m & 3)*FPS;
                plane(SU, u, lo4, so); plane(SV, v, lo4, so); plane(SW, w, lo4, so);
                if (DIF) plane(SE, ev, lo4, so);
                if (SCAL) plane(SS, s, (unsigned)(m + 3)*ij, ((m + 3) & 3)*FPS);
            }
            cp_async_commit();

            if (write)
            {
                const int gx0 = gxi, gy0 = gyi;
                const TF zf = pl[5*PLEV - 1];
                if constexpr (sizeof(TF) == 4)
                {
                    // The four fields' face fluxes in one 16-byte load per face;
                    // u/v and w/s in packed pairs.
                    const float4 xa = reinterpret_cast<const float4*>(gx)[gx0];
                    const float4 xb = reinterpret_cast<const float4*>(gx)[gx0 + 1];
                    const float4 ya = reinterpret_cast<const float4*>(gy)[gy0];
                    const float4 yb = reinterpret_cast<const float4*>(gy)[gy0 + FTX];
                    {
                        const float2 dgx = sub2(f2(xb.x, xb.y), f2(xa.x, xa.y));
                        const float2 dgy = sub2(f2(yb.x, yb.y), f2(ya.x, ya.y));
                        const float2 dgz = sub2(f2(gzu_t, gzv_t), f2(gzu_b, gzv_b));
                        const float2 t = __ffma2_rn(dgz, f2(zf, zf), __ffma2_rn(dgy, f2(dyi, dyi),
                                                    __ffma2_rn(dgx, f2(dxi, dxi), f2(tu, tv))));
                        a.ut[c] = t.x; a.vt[c] = t.y;
                    }
                    if constexpr (SCAL)
                    {
                        const float2 dgx = sub2(f2(xb.z, xb.w), f2(xa.z, xa.w));
                        const float2 dgy = sub2(f2(yb.z, yb.w), f2(ya.z, ya.w));
                        const float2 dgz = sub2(f2(gzw_t, gzs_t), f2(gzw_b, gzs_b));
                        const float2 t = __ffma2_rn(dgz, f2(pl[6*PLEV], zf), __ffma2_rn(dgy, f2(dyi, dyi),
                                                    __ffma2_rn(dgx, f2(dxi, dxi), f2(tw + buoy, ts))));
                        if (wlev) a.wt[c + ij] = t.x;
                        a.st[c] = t.y;
                    }
                    else if (wlev)
                        a.wt[c + ij] = tw + (xb.z - xa.z)*dxi + (yb.z - ya.z)*dyi
                                                 + (gzw_t - gzw_b)*pl[6*PLEV] + buoy;
                }
                else
                {
                    a.ut[c] = tu + (gx[(gx0 + 1)*4 + 0] - gx[(gx0)*4 + 0])*dxi
                                 + (gy[(gy0 + FTX)*4 + 0] - gy[(gy0)*4 + 0])*dyi + (gzu_t - gzu_b)*zf;
                    a.vt[c] = tv + (gx[(gx0 + 1)*4 + 1] - gx[(gx0)*4 + 1])*dxi
                                 + (gy[(gy0 + FTX)*4 + 1] - gy[(gy0)*4 + 1])*dyi + (gzv_t - gzv_b)*zf;
                    if (wlev)
                        a.wt[c + ij] = tw + (gx[(gx0 + 1)*4 + 2] - gx[(gx0)*4 + 2])*dxi
                                                 + (gy[(gy0 + FTX)*4 + 2] - gy[(gy0)*4 + 2])*dyi
                                                 + (gzw_t - gzw_b)*pl[6*PLEV] + buoy;
                    if (SCAL)
                        a.st[c] = ts + (gx[(gx0 + 1)*4 + 3] - gx[(gx0)*4 + 3])*dxi
                                     + (gy[(gy0 + FTX)*4 + 3] - gy[(gy0)*4 + 3])*dyi + (gzs_t - gzs_b)*zf;
                }
            }

            gzu_b = gzu_t; gzv_b = gzv_t; gzw_b = gzw_t; gzs_b = gzs_t;
            ex0 = ex1; ey0 = ey1;
            #pragma unroll
            for (int q=0; q<5; ++q) { qu[q] = qu[q+1]; qv[q] = qv[q+1]; qw[q] = qw[q+1]; qs[q] = qs[q+1]; }
            qu[5] = nu; qv[5] = nv; qw[5] = nw; qs[5] = ns;
        }
        cp_async_wait_all();
    }

    template<typename TF, bool SURF, bool SCAL, bool BUOY, bool LIM = false, bool ADV = true, bool DIF = true>
    static void launch_flux_t(const Dims& d, const Prof<TF>& pr, const TendArgs<TF>& a, int kchunk, cudaStream_t s)
    {
        const size_t smem = flux_smem<TF>();
        kchunk = auto_kchunk(kchunk, (long long)((d.itot + FTX - 1)/FTX)*((d.jtot + FTY - 1)/FTY), d.ktot,
                             sizeof(TF) == 8, FKCHUNK_MAX);
        dim3 grid((d.itot + FTX - 1)/FTX, (d.jtot + FTY - 1)/FTY, (d.ktot + kchunk - 1)/kchunk);
        launch_body<TendFluxP<TF>, tend_flux_body<TF, SURF, SCAL, BUOY, LIM, ADV, DIF>, NTHR, FluxOcc<TF>::v>(
            grid, dim3(NTHR), smem, s, TendFluxP<TF>{d, pr, a, kchunk});
        count_launch();
    }

    // Advec_2i5 + Diff_smag2 (+ buoyancy) in flux form; igc, jgc >= 3.
    template<typename TF>
    void launch_tendency_flux(const Dims& d, const Prof<TF>& pr, const TendArgs<TF>& a, bool surf, bool scal,
                              bool buoy, bool lim, int kchunk, cudaStream_t s)
    {
        if (lim && scal)
        {
            if (surf && buoy) launch_flux_t<TF, true, true, true, true>(d, pr, a, kchunk, s);
            else if (surf) launch_flux_t<TF, true, true, false, true>(d, pr, a, kchunk, s);
            else if (buoy) launch_flux_t<TF, false, true, true, true>(d, pr, a, kchunk, s);
            else launch_flux_t<TF, false, true, false, true>(d, pr, a, kchunk, s);
            return;
        }
        const int mask = (surf ? 4 : 0) | (scal ? 2 : 0) | (buoy ? 1 : 0);
        switch (mask)
        {
            case 0: launch_flux_t<TF, false, false, false>(d, pr, a, kchunk, s); break;
            case 1: launch_flux_t<TF, false, false, true >(d, pr, a, kchunk, s); break;
            case 2: launch_flux_t<TF, false, true,  false>(d, pr, a, kchunk, s); break;
            case 3: launch_flux_t<TF, false, true,  true >(d, pr, a, kchunk, s); break;
            case 4: launch_flux_t<TF, true,  false, false>(d, pr, a, kchunk, s); break;
            case 5: launch_flux_t<TF, true,  false, true >(d, pr, a, kchunk, s); break;
            case 6: launch_flux_t<TF, true,  true,  false>(d, pr, a, kchunk, s); break;
            default: launch_flux_t<TF, true, true,  true >(d, pr, a, kchunk, s); break;
        }
    }

    template<typename TF>
    void launch_tendency_flux_term(const Dims& d, const Prof<TF>& pr, const TendArgs<TF>& a, bool adv, bool surf,
                                   bool scal, bool lim, int kchunk, cudaStream_t s)
    {
        if (adv)
        {
            if (lim && scal) launch_flux_t<TF, false, true, false, true, true, false>(d, pr, a, kchunk, s);
            else if (scal) launch_flux_t<TF, false, true, false, false, true, false>(d, pr, a, kchunk, s);
            else launch_flux_t<TF, false, false, false, false, true, false>(d, pr, a, kchunk, s);
        }
        else if (surf)
        {
            if (scal) launch_flux_t<TF, true, true, false, false, false, true>(d, pr, a, kchunk, s);
            else launch_flux_t<TF, true, false, false, false, false, true>(d, pr, a, kchunk, s);
        }
        else
        {
            if (scal) launch_flux_t<TF, false, true, false, false, false, true>(d, pr, a, kchunk, s);
            else launch_flux_t<TF, false, false, false, false, false, true>(d, pr, a, kchunk, s);
        }
    }

    template void launch_tendency_flux_term<double>(const Dims&, const Prof<double>&, const TendArgs<double>&, bool, bool, bool, bool, int, cudaStream_t);
    template void launch_tendency_flux_term<float>(const Dims&, const Prof<float>&, const TendArgs<float>&, bool, bool, bool, bool, int, cudaStream_t);
    template void launch_tendency_flux<double>(const Dims&, const Prof<double>&, const TendArgs<double>&, bool, bool, bool, bool, int, cudaStream_t);
    template void launch_tendency_flux<float>(const Dims&, const Prof<float>&, const TendArgs<float>&, bool, bool, bool, bool, int, cudaStream_t);
}
