// mhh_surface.cu -- Monin-Obukhov surface layer on the GPU, after
// src/boundary_surface.cxx:836-994 and include/boundary_surface_kernels.h
// (lookup-table Obukhov-length solver with homogeneous z0m/z0h, noslip
// momentum, flux or Dirichlet scalar).  The 2-D fields are stored in double;
// the Obukhov length and the similarity functions are computed in the field
// precision (double for the FP64 path, float for the FP32 form, which keeps
// the float form off the slow FP64 pipe).  The z/L lookup table and the
// Richardson-number interpolation stay in float as in the reference, with the
// float operations rounded one by one so that they match the CPU bit for bit.
#include "mhh_kernels.cuh"
#include "mhh_batchable.cuh"

namespace mhh
{
    // Monin-Obukhov similarity functions, include/monin_obukhov.h:40-152, in
    // the compute type CT (double for the FP64 path, float for the FP32 form).
    template<typename CT> __device__ __forceinline__ CT phim_unstable(CT z)
    { return pow(CT(1) + CT(3.6)*pow(fabs(z), CT(2./3.)), CT(-1./2.)); }
    template<typename CT> __device__ __forceinline__ CT phih_unstable(CT z)
    { return pow(CT(1) + CT(7.9)*pow(fabs(z), CT(2./3.)), CT(-1./2.)); }
    template<typename CT> __device__ __forceinline__ CT phim(CT z) { return z <= CT(0) ? phim_unstable(z) : CT(1) + CT(5)*z; }
    template<typename CT> __device__ __forceinline__ CT phih(CT z) { return z <= CT(0) ? phih_unstable(z) : (CT(1) + CT(4)*z)*(CT(1) + CT(4)*z); }
    template<typename CT> __device__ __forceinline__ CT psim_stable(CT z)
    {
        const CT a = 1, b = CT(2)/CT(3), c = 5, d = CT(0.35);
        return -b*(z - (c/d))*exp(-d*z) - a*z - (b*c)/d;
    }
    template<typename CT> __device__ __forceinline__ CT psih_stable(CT z)
    {
        const CT a = 1, b = CT(2)/CT(3), c = 5, d = CT(0.35);
        return -b*(z - (c/d))*exp(-d*z) - pow(CT(1) + b*a*z, CT(1.5)) - (b*c)/d + CT(1);
    }

    // include/boundary_surface_kernels.h:282-298, with the search kept inside
    // the table.  The walk from the cell's last position reads eight entries
    // at a time, so that it waits once per eight steps (the first call walks
    // from the bottom of the table).
    __device__ double find_zL(const float* __restrict__ zL, const float* __restrict__ f, int* np, float Ri)
    {
        constexpr int W = 8;
        int n = *np;
        if (__fsub_rn(f[n], Ri) > 0.f)
        {
            for (bool more = true; more && n > 0; )
            {
                float v[W];
                #pragma unroll
                for (int q=0; q<W; ++q) v[q] = f[max(n - 1 - q, 0)];
                #pragma unroll
                for (int q=0; q<W; ++q)
                {
                    more = more && n > 0 && __fsub_rn(v[q], Ri) > 0.f;
                    if (more) --n;
                }
            }
        }
        else
        {
            for (bool more = true; more && n < NZL_LUT-1; )
            {
                float v[W];
                #pragma unroll
                for (int q=0; q<W; ++q) v[q] = f[min(n + q, NZL_LUT - 1)];
                #pragma unroll
                for (int q=0; q<W; ++q)
                {
                    more = more && __fsub_rn(v[q], Ri) < 0.f && n < NZL_LUT-1;
                    if (more) ++n;
                }
            }
        }
        *np = n;
        if (n == 0 || n == NZL_LUT-1) return (double)zL[n];
        const float num = __fsub_rn(Ri, f[n-1]);
        const float den = __fsub_rn(f[n], f[n-1]);
        const float dz = __fsub_rn(zL[n], zL[n-1]);
        return (double)__fadd_rn(zL[n-1], __fmul_rn(__fdiv_rn(num, den), dz));
    }

    // Everything the surface-layer kernels of one context read and write.
    template<typename TF> struct SurfP
    {
        Dims d; SurfWork sw;
        const TF *u, *v, *s;
        TF *u_bot, *v_bot, *u_flux, *v_flux, *u_grad, *v_grad, *s_bot, *s_flux, *s_grad;
        double zsl, z0m, z0h, thref_s, threfh_s, thb_s, thbh_s;
        int thermo, thermo_bc;
        SurfGhost<TF> g;
    };

    // Filtered wind speed of the interior cell ij,
    // include/boundary_surface_kernels.h:132-178, in the field precision.
    template<typename TF>
    __device__ __forceinline__ TF wind_speed(const SurfP<TF>& P, int ij)
    {
        const Dims& d = P.d;
        const TF* __restrict__ u = P.u; const TF* __restrict__ v = P.v;
        const TF* __restrict__ ubot = P.u_bot; const TF* __restrict__ vbot = P.v_bot;
        const long long ii = 1, jj = d.icells;
        const long long c = ij + (long long)d.kstart*d.ijcells;
        using CT = TF;
        auto U = [&](long long q) { return CT(u[q]); };
        auto V = [&](long long q) { return CT(v[q]); };
        const CT h = CT(0.5);
        const CT uf = CT(1./9)*(
              h*U(c-ii-jj) + U(c-jj) + U(c+ii-jj) + h*U(c+2*ii-jj)
            + h*U(c-ii   ) + U(c   ) + U(c+ii   ) + h*U(c+2*ii   )
            + h*U(c-ii+jj) + U(c+jj) + U(c+ii+jj) + h*U(c+2*ii+jj));
        const CT vf = CT(1./9)*(
              h*V(c-ii-jj) + V(c-ii) + V(c-ii+jj) + h*V(c-ii+2*jj)
            + h*V(c   -jj) + V(c   ) + V(c   +jj) + h*V(c   +2*jj)
            + h*V(c+ii-jj) + V(c+ii) + V(c+ii+jj) + h*V(c+ii+2*jj));
        const CT du2 = sq(uf - h*(CT(ubot[ij]) + CT(ubot[ij+ii])))
                     + sq(vf - h*(CT(vbot[ij]) + CT(vbot[ij+jj])));
        return fmax(pow(du2, CT(0.5)), CT(1.e-1));
    }

    // The Monin-Obukhov functions of one cell, each evaluated once: the
    // similarity function phi of the stability branch feeds both the
    // integrated psi and the gradient (include/monin_obukhov.h:40-152).
    template<typename CT> struct MostCell { CT fm, fh, phim, phih; };

    template<typename CT>
    __device__ __forceinline__ MostCell<CT> most_cell(CT zsl, CT z0m, CT z0h, CT L)
    {
        MostCell<CT> r;
        const CT kappa = CT(KAPPA);
        const CT zeta = zsl/L;
        if (L <= CT(0))
        {
            const CT pm_s = phim_unstable(zeta), pm_0 = phim_unstable(z0m/L);
            const CT ph_s = phih_unstable(zeta), ph_0 = phih_unstable(z0h/L);
            const CT psim_s = CT(3)*log((CT(1) + CT(1)/pm_s)/CT(2)), psim_0 = CT(3)*log((CT(1) + CT(1)/pm_0)/CT(2));
            const CT psih_s = CT(3)*log((CT(1) + CT(1)/ph_s)/CT(2)), psih_0 = CT(3)*log((CT(1) + CT(1)/ph_0)/CT(2));
            r.fm = kappa/(log(zsl/z0m) - psim_s + psim_0);
            r.fh = kappa/(log(zsl/z0h) - psih_s + psih_0);
            r.phim = zeta <= CT(0) ? pm_s : CT(1) + CT(5)*zeta;
            r.phih = zeta <= CT(0) ? ph_s : (CT(1) + CT(4)*zeta)*(CT(1) + CT(4)*zeta);
        }
        else
        {
            r.fm = kappa/(log(zsl/z0m) - psim_stable(zeta) + psim_stable(z0m/L));
            r.fh = kappa/(log(zsl/z0h) - psih_stable(zeta) + psih_stable(z0h/L));
            r.phim = phim(zeta);
            r.phih = phih(zeta);
        }
        return r;
    }

    // The surface layer runs as two kernels over all cells of the 2-D arrays,
    // ghost cells included: the Obukhov state of every cell, then everything
    // that needs its neighbours'; a ghost cell computes its image's values from
    // the same operands, which equals the periodic copy of the reference.  One
    // kernel per module of the reference and per periodic copy made nine
    // launches, bound by launch and latency: per RK3 step with the scalar's ghost
    // levels 0.125 ms at 32^3 and 0.19 at 512 x 512, now 0.049 and 0.11; in double
    // 0.36 at 64^3, now 0.15.
    constexpr int SURF_NT = 64;

    // Wind speed, Obukhov length and friction velocity,
    // src/boundary_surface.cxx:55-160 (the neutral branch when there is no
    // thermodynamics).  Blocks of two warps: a double evaluation of the
    // similarity functions is some 300 operations on the narrow FP64 pipe, so
    // small grids spread over all SMs.
    template<typename TF>
    __device__ __forceinline__ void surf_state_body(const SurfP<TF>& P, const VBlock& vb)
    {
        const Dims& d = P.d;
        const SurfWork& sw = P.sw;
        const TF* __restrict__ s = P.s; const TF* __restrict__ s_bot = P.s_bot; const TF* __restrict__ s_flux = P.s_flux;
        const double zsl = P.zsl, z0m = P.z0m, thref_s = P.thref_s, threfh_s = P.threfh_s;
        const double thb_s = P.thb_s, thbh_s = P.thbh_s;
        const int thermo = P.thermo, thermo_bc = P.thermo_bc;
        const int n = vb.x*blockDim.x + threadIdx.x;
        if (n >= d.ijcells) return;
        using CT = TF;
        bool inside;
        const CT du = wind_speed(P, plane_image(d, n, inside));
        const CT zs = CT(zsl);
        CT L;
        if (!thermo)
            L = CT(-DBIG);
        else if (thermo_bc == MHH_BC_FLUX)
        {
            const CT bfluxbot = CT(GRAV)/CT(threfh_s)*CT(s_flux[n]);
            const float Ri = (float)(CT(-KAPPA)*bfluxbot*zs/(du*du*du));
            L = zs/CT(find_zL(sw.zL, sw.f, &sw.nobuk[n], Ri));
        }
        else
        {
            // theta - thref in the scalar's storage units (thb = thref - offset).
            const CT b = CT(GRAV)/CT(thref_s)*(CT(s[n + (long long)d.kstart*d.ijcells]) - CT(thb_s));
            const CT bbot = CT(GRAV)/CT(threfh_s)*(CT(s_bot[n]) - CT(thbh_s));
            const CT db_ref = CT(GRAV)/CT(thref_s)*(CT(thref_s) - CT(threfh_s));
            const CT db = b - bbot + db_ref;
            const float Ri = (float)(CT(KAPPA)*db*zs/(du*du));
            L = zs/CT(find_zL(sw.zL, sw.f, &sw.nobuk[n], Ri));
        }
        const MostCell<CT> mc = most_cell<CT>(zs, CT(z0m), CT(sw.z0h), L);
        sw.obuk[n] = to_d<CT>(L);
        sw.ustar[n] = to_d<CT>(du*mc.fm);
        sw.fm[n] = to_d<CT>(mc.fm); sw.fh[n] = to_d<CT>(mc.fh);
        sw.phim[n] = to_d<CT>(mc.phim); sw.phih[n] = to_d<CT>(mc.phih);
    }

    // Momentum fluxes (src/boundary_surface.cxx:163-190), surface gradients of
    // u and v and the scalar's surface value, gradient or flux (:255-338), the
    // Monin-Obukhov gradients for the next viscosity (interior cells,
    // include/boundary_surface_kernels.h:180-238) and, where the caller asks,
    // the scalar's wall ghost levels.
    template<typename TF>
    __device__ __forceinline__ void surf_flux_body(const SurfP<TF>& P, const VBlock& vb)
    {
        const Dims& d = P.d;
        const SurfWork& sw = P.sw;
        const TF* __restrict__ u = P.u; const TF* __restrict__ v = P.v; const TF* s = P.s;
        const TF* __restrict__ ubot = P.u_bot; const TF* __restrict__ vbot = P.v_bot;
        const double zsl = P.zsl, threfh_s = P.threfh_s;
        const int thermo = P.thermo, thermo_bc = P.thermo_bc;
        const int n = vb.x*blockDim.x + threadIdx.x;
        if (n >= d.ijcells) return;
        bool inside;
        const int ij = plane_image(d, n, inside);
        const int ii = 1, jj = d.icells;
        const long long k0 = (long long)d.kstart*d.ijcells;
        using CT = TF;
        auto D = [&](const double* a, int q) { return from_d<CT>(a[q]); };
        {
            const CT fc = D(sw.ustar, ij)*D(sw.fm, ij);
            P.u_flux[n] = -(CT(u[k0 + ij]) - CT(ubot[ij]))*CT(0.5)*(D(sw.ustar, ij-ii)*D(sw.fm, ij-ii) + fc);
            P.v_flux[n] = -(CT(v[k0 + ij]) - CT(vbot[ij]))*CT(0.5)*(D(sw.ustar, ij-jj)*D(sw.fm, ij-jj) + fc);
        }
        const CT z = CT(zsl);
        P.u_grad[n] = (CT(u[k0 + n]) - CT(ubot[n]))/z;
        P.v_grad[n] = (CT(v[k0 + n]) - CT(vbot[n]))/z;
        CT flux = CT(0);
        if (thermo)
        {
            const CT th = CT(s[k0 + n]);
            const CT us = from_d<CT>(sw.ustar[n]), fh = from_d<CT>(sw.fh[n]);
            flux = CT(P.s_flux[n]);
            if (thermo_bc == MHH_BC_DIRICHLET)
            {
                flux = -(th - CT(P.s_bot[n]))*us*fh;
                P.s_flux[n] = flux;
                P.s_grad[n] = (th - CT(P.s_bot[n]))/z;
            }
            else
            {
                const CT bot = flux/(us*fh) + th;
                P.s_bot[n] = bot;
                P.s_grad[n] = (th - bot)/z;
            }
        }
        if (inside)
        {
            const long long c = k0 + n;
            const CT du_c = CT(0.5)*((CT(u[c]) - CT(ubot[n])) + (CT(u[c+ii]) - CT(ubot[n+ii])));
            const CT dv_c = CT(0.5)*((CT(v[c]) - CT(vbot[n])) + (CT(v[c+jj]) - CT(vbot[n+jj])));
            const CT us = from_d<CT>(sw.ustar[n]);
            const CT fmv = from_d<CT>(sw.fm[n]);
            const CT ufb = -du_c*us*fmv;
            const CT vfb = -dv_c*us*fmv;
            const CT ph = from_d<CT>(sw.phim[n]);
            const CT kz = CT(KAPPA)*CT(zsl);
            sw.dudz[n] = to_d<CT>(-ufb/(kz*us)*ph);
            sw.dvdz[n] = to_d<CT>(-vfb/(kz*us)*ph);
            if (thermo)
            {
                const CT bfb = CT(GRAV)/CT(threfh_s)*flux;
                sw.dbdz[n] = to_d<CT>(-bfb/(kz*us)*from_d<CT>(sw.phih[n]));
            }
        }
        if (P.g.a)
        {
            const SurfGhost<TF>& g = P.g;
            const long long cb = k0 + n, ct = n + (long long)(d.kend-1)*d.ijcells;
            wall_ghost(g.a, n, cb, ct, d.ijcells, g.bot_type, g.bot, g.gradbot, g.dzh[d.kstart],
                       g.top_type, g.top, g.gradtop, g.dzh[d.kend]);
        }
    }

    template<typename TF>
    void launch_surface(const Dims& d, const Prof<TF>& pr, const SurfWork& sw,
                        const TF* u, const TF* v, const TF* s,
                        TF* u_bot, TF* v_bot, TF* u_flux, TF* v_flux, TF* u_grad, TF* v_grad,
                        TF* s_bot, TF* s_flux, TF* s_grad,
                        int thermo, int thermo_bc, double z0m, double z0h, const SurfGhost<TF>& ghost, cudaStream_t st)
    {
        const double zsl = sw.zsl, thref_s = sw.thref_s, threfh_s = sw.threfh_s;
        const dim3 nb((d.ijcells + SURF_NT - 1)/SURF_NT);
        const SurfP<TF> P{d, sw, u, v, s, u_bot, v_bot, u_flux, v_flux, u_grad, v_grad, s_bot, s_flux, s_grad,
                          zsl, z0m, z0h, thref_s, threfh_s, sw.thb_s, sw.thbh_s, thermo, thermo_bc, ghost};
        launch_body<SurfP<TF>, surf_state_body<TF>, SURF_NT>(nb, dim3(SURF_NT), 0, st, P);
        launch_body<SurfP<TF>, surf_flux_body<TF>, SURF_NT>(nb, dim3(SURF_NT), 0, st, P);
        count_launch(2);
    }

    template void launch_surface<double>(const Dims&, const Prof<double>&, const SurfWork&, const double*, const double*,
        const double*, double*, double*, double*, double*, double*, double*, double*, double*, double*,
        int, int, double, double, const SurfGhost<double>&, cudaStream_t);
    template void launch_surface<float>(const Dims&, const Prof<float>&, const SurfWork&, const float*, const float*,
        const float*, float*, float*, float*, float*, float*, float*, float*, float*, float*,
        int, int, double, double, const SurfGhost<float>&, cudaStream_t);
}
