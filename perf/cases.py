"""The work this framework's users give it, as measured cases.

Each case is one call of the public API on a model (or an ensemble of models)
whose state lives on the GPU: RK3 time steps of the dry convective boundary
layer (Advec_2i5, Smagorinsky, Monin-Obukhov surface, Pres_2) and of the
turbulent channel (Advec_2, Diff_2, Pres_2), in the FP32 form and in the plain
FP64 path, from the smallest grids of the ensembles and the serving loop to the
512 x 512 x 256 benchmark.

    listed()             the cases
    draw(rng)            one more case of the same ranges
    prepare(case, seed)  models and their initial state on the GPU
    run(state)           one pass, and the fields it leaves
    work(case)           bytes and operations of one pass
    exact(case, seed)    the same fields in 64 bits, in plain torch

The initial states are those of a running simulation: a boundary layer with a
mean wind, solenoidal eddies of about 1 m/s and theta noise in the lowest
levels; for the channel the laminar profile with 5% Gaussian noise.
"""
import math

import numpy as np
import torch

import microhh_gb300 as mhh
from microhh_gb300 import cases as mcases

THREF = 300.0
GRAV = 9.81
KAPPA = 0.4
CB = (1. / 3., 15. / 16., 8. / 15.)
CA = (0., -5. / 9., -153. / 128.)

# The grids of the ensemble workload.
MEMBER_GRIDS = ((32, 32, 32), (48, 48, 64), (64, 64, 64), (96, 96, 64), (128, 128, 96))


def listed():
    return [
        # The smallest member of an ensemble, the smallest served job: bound by
        # launches and latency.
        les("les_f32_32x32x32", 32, 32, 32, 32),
        # The parity configuration in the plain FP64 path.
        les("les_f64_64x64x64", 64, 64, 64, 64),
        # The largest ensemble member.
        les("les_f32_128x128x96", 32, 128, 128, 96),
        # A served job whose sides have the factors 3 and 5.
        les("les_f32_150x150x150", 32, 150, 150, 150),
        # Odd sides and ragged tiles, with the two options a boundary-layer run
        # turns on in earnest: a damping layer and the limited scalar.
        les("les_options_f32_189x105x90", 32, 189, 105, 90, options=True),
        # The reference's module order, one call per module, as a host that
        # binds the modules one by one runs it.
        les("les_modules_f32_96x96x64", 32, 96, 96, 64, fused=False),
        # A monitored run: a step, then the CFL number and the profiles.
        les("les_monitored_f32_256x256x128", 32, 256, 256, 128, monitored=True),
        # The plain FP64 path on an ordinary large grid.
        les("les_f64_256x256x128", 64, 256, 256, 128),
        # The benchmark.
        les("les_f32_512x512x256", 32, 512, 512, 256),
        # The channel configuration in both precisions, with its adaptive step.
        channel("channel_f32_256x192x128", 32, 256, 192, 128),
        channel("channel_f64_256x192x128", 64, 256, 192, 128),
        # Members of uneven sizes advanced together through CUDA graphs.
        ensemble("ensemble_f32_12", 12, 0),
    ]


def les(name, prec, itot, jtot, ktot, options=False, fused=True, monitored=False):
    c = {"kind": "les", "prec": prec, "itot": itot, "jtot": jtot, "ktot": ktot,
         "options": options, "fused": fused, "monitored": monitored}
    return dict(c, name=name) if name else c


def channel(name, prec, itot, jtot, ktot):
    c = {"kind": "channel", "prec": prec, "itot": itot, "jtot": jtot, "ktot": ktot}
    return dict(c, name=name) if name else c


def ensemble(name, members, first):
    c = {"kind": "ensemble", "prec": 32, "members": members, "first": first, "steps": 2}
    return dict(c, name=name) if name else c


def smooth(lo, hi):
    """Lengths the transforms take (2^a 3^b 5^c 7^d), odd ones among them."""
    out = []
    for n in range(lo, hi + 1):
        r = n
        for f in (2, 3, 5, 7):
            while r % f == 0:
                r //= f
        if r == 1:
            out.append(n)
    return out


def pick(rng, lo, hi):
    """A transform length, log-uniform."""
    t = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return min(smooth(lo, hi), key=lambda n: abs(math.log(n / t)))


def levels(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["les32", "les32", "les32", "les64", "options", "modules", "monitored",
                       "channel32", "channel64", "ensemble"])
    if kind == "les32":
        return les(None, 32, pick(rng, 24, 512), pick(rng, 24, 512), levels(rng, 24, 256))
    if kind == "les64":
        return les(None, 64, pick(rng, 24, 256), pick(rng, 24, 256), levels(rng, 24, 128))
    if kind == "options":
        return les(None, 32, pick(rng, 32, 256), pick(rng, 32, 256), levels(rng, 24, 128), options=True)
    if kind == "modules":
        return les(None, rng.choice([32, 64]), pick(rng, 24, 160), pick(rng, 24, 160), levels(rng, 24, 96), fused=False)
    if kind == "monitored":
        return les(None, 32, pick(rng, 48, 384), pick(rng, 48, 384), levels(rng, 24, 192), monitored=True)
    if kind == "ensemble":
        return ensemble(None, rng.randint(4, 15), rng.randrange(1 << 16))
    prec = 32 if kind == "channel32" else 64
    return channel(None, prec, pick(rng, 32, 256), pick(rng, 24, 192), levels(rng, 24, 128))


# ---------------------------------------------------------------------------
# Set-up
# ---------------------------------------------------------------------------
def sizes(case):
    """(itot, jtot, ktot, surface flux, lapse rate) of every model of a case."""
    if case["kind"] != "ensemble":
        return [(case["itot"], case["jtot"], case["ktot"], 0.1, 0.003)]
    out = []
    for m in range(case["members"]):
        g = MEMBER_GRIDS[(m + case["first"]) % len(MEMBER_GRIDS)]
        out.append(g + (0.05 + 0.2 * ((7 * m + 3) % 11) / 10., 0.001 + 0.005 * ((5 * m + 1) % 7) / 6.))
    return out


def setup(case, itot, jtot, ktot, sbot, lapse):
    """The model description (without fields) of one grid of the case."""
    if case["kind"] == "channel":
        return mcases.Case(
            name="channel", itot=itot, jtot=jtot, ktot=ktot, xsize=2. * math.pi, ysize=math.pi, zsize=2.,
            z=mcases.stretched_channel_z(ktot, 2.75), advec="2", diff="2", thermo=False, surface=False,
            mbcbot=mcases.BC_DIRICHLET, mbctop=mcases.BC_DIRICHLET, sbcbot=mcases.BC_FLUX, sbctop=mcases.BC_FLUX,
            sbot=0., stop=0., visc=1. / 180., svisc=1. / 180., swlspres=True, dpdx=-1., dt=1.e-3, adaptivestep=True)
    dx = 100. if case["kind"] == "ensemble" else 50.
    c = mcases.Case(
        name="drycbl", itot=itot, jtot=jtot, ktot=ktot, xsize=dx * itot, ysize=dx * jtot, zsize=4000.,
        z=mcases.uniform_z(ktot, 4000.), sbot=sbot, stop=lapse, dt=2.)
    if case.get("options"):
        c.swbuffer, c.buffer_zstart, c.buffer_sigma, c.buffer_beta = True, 3000., 0.01, 2.
        c.fluxlimit = True
    return c


def initial(case, c, seed):
    """The initial fields on the GPU in double: {name: (ktot, jtot, itot)}."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed)
    f8 = dict(dtype=torch.float64, device=dev)
    sh = (c.ktot, c.jtot, c.itot)
    z = torch.as_tensor(np.asarray(c.z), **f8)
    if case["kind"] == "channel":
        ub = 15.6
        u = (1.5 * ub * (1. - (z - 1.) ** 2))[:, None, None] + 0.05 * ub * torch.randn(sh, generator=gen, **f8)
        v = 0.05 * ub * torch.randn(sh, generator=gen, **f8)
        w = 0.05 * ub * torch.randn(sh, generator=gen, **f8)
        w[0] = 0.
        return {"u": u, "v": v, "w": w}

    # Eddies: the discrete curl of a potential of a few modes that vanish at
    # the walls, so that the divergence is zero on the staggered grid.
    rnd = np.random.RandomState(seed % (1 << 32))
    nm = 6
    dz = c.zsize / c.ktot
    dx, dy = c.xsize / c.itot, c.ysize / c.jtot

    def potential(xo, yo, zo, n):
        """Sum of modes at offsets (in cells) of the grid, n levels."""
        x = (torch.arange(c.itot, **f8) + xo) * (2. * math.pi / c.itot)
        y = (torch.arange(c.jtot, **f8) + yo) * (2. * math.pi / c.jtot)
        zz = (torch.arange(n, **f8) + zo) * (math.pi / c.ktot)
        t = lambda a: torch.as_tensor(a, **f8)[:, None]  # noqa: E731
        a = torch.cos(t(rnd.randint(1, 5, nm)) * x + t(rnd.uniform(0, 6.28, nm)))
        b = torch.cos(t(rnd.randint(1, 5, nm)) * y + t(rnd.uniform(0, 6.28, nm)))
        q = torch.sin(t(rnd.randint(1, 4, nm)) * zz) * t(rnd.uniform(0.5, 1., nm))
        q[:, 0] = 0. if zo == 0 else q[:, 0]
        if n == c.ktot + 1:
            q[:, -1] = 0.
        return torch.einsum("mk,mj,mi->kji", q, b, a)

    ax = potential(0.5, 0., 0., c.ktot + 1)
    ay = potential(0., 0.5, 0., c.ktot + 1)
    az = potential(0., 0., 0.5, c.ktot)
    right = lambda a, d: torch.roll(a, -1, d)  # noqa: E731
    u = (right(az, 1) - az) / dy - (ay[1:] - ay[:-1]) / dz
    v = (ax[1:] - ax[:-1]) / dz - (right(az, 2) - az) / dx
    w = ((right(ay, 2) - ay) / dx - (right(ax, 1) - ax) / dy)[:c.ktot]
    s = 1. / max(float(u.std()), float(v.std()), float(w.std()))
    u, v, w = 2. + s * u, -1. + s * v, s * w
    w[0] = 0.
    th = torch.where(z < 1000., THREF + 0. * z, THREF + c.stop * (z - 1000.))[:, None, None].repeat(1, c.jtot, c.itot)
    low = max(1, int((z < 400.).sum()))
    th[:low] += 0.2 * torch.rand((low,) + sh[1:], generator=gen, **f8) - 0.1
    return {"u": u, "v": v, "w": w, "th": th}


def stored(case, fields):
    """The fields as the model stores them: in the FP32 form float, with theta
    as its difference from the reference temperature."""
    if case["prec"] == 64:
        return fields
    return {n: (a - THREF if n == "th" else a).to(torch.float32) for n, a in fields.items()}


class Device:
    """A device field for torch.as_tensor: the tensor made from it holds this
    object and with it the model that owns the memory."""

    def __init__(self, model, ptr):
        self.model = model
        self.__cuda_array_interface__ = {"shape": model.shape, "typestr": "<f8" if model.precision == 64 else "<f4",
                                         "data": (ptr, False), "version": 3, "strides": None}


def interior(model, c, ptr):
    """A view of the interior cells of a device field."""
    a = torch.as_tensor(Device(model, ptr), device="cuda")
    g, k = c.igc, c.kgc
    return a[k:k + c.ktot, g:g + c.jtot, g:g + c.itot]


def make_model(case, c, seed):
    """A model with its initial state, and views of the fields it steps (and
    of p; the channel's p after a projected step is the round-off of u/dt)."""
    m = mhh.Model(ini=c.to_ini(), z=c.z, precision=case["prec"])
    f, _ = m.device_fields()
    ptr = {"u": f.u, "v": f.v, "w": f.w, "th": f.s, "p": f.p}
    ini = initial(case, c, seed)
    if c.swbuffer:
        for n in ("u", "v", "th"):
            prof = np.zeros(c.ktot + 2 * c.kgc)
            prof[c.kgc:c.kgc + c.ktot] = ini[n].mean(dim=(1, 2)).cpu().numpy()
            m.set_buffer_profile(n, prof)
    ini = stored(case, ini)
    names = ("u", "v", "w", "th") if c.thermo else ("u", "v", "w")
    for n in names:
        interior(m, c, ptr[n]).copy_(ini[n])
    out = {n: interior(m, c, ptr[n]) for n in names + (("p",) if case["kind"] == "les" else ())}
    return m, out


def prepare(case, seed):
    models, outs = [], []
    for q, (itot, jtot, ktot, sbot, lapse) in enumerate(sizes(case)):
        m, out = make_model(case, setup(case, itot, jtot, ktot, sbot, lapse), seed + 1000 * q)
        models.append(m)
        outs.append(out)
    torch.cuda.synchronize()
    if case["kind"] == "ensemble":
        return {"ens": mhh.Ensemble(models), "models": models, "out": outs, "steps": case["steps"]}
    return {"model": models[0], "out": outs[0], "fused": case.get("fused", True), "monitored": case.get("monitored", False)}


# ---------------------------------------------------------------------------
# The pass
# ---------------------------------------------------------------------------
def run(state):
    if "ens" in state:
        state["ens"].run_steps(state["steps"], mhh.ENS_GRAPHS)
        return state["out"]
    m = state["model"]
    m.run_steps(1, fused=state["fused"])
    if not state["monitored"]:
        return state["out"]
    out = dict(state["out"], cfl=np.float64(m.cfl()))
    # The levels of the domain (the profiles come with the ghost levels).
    for n in ("u", "v", "th"):
        mean, var = m.profile_stats(n)
        out[n + "_mean"], out[n + "_var"] = mean[1:-1], var[1:-1]
    out["w_var"] = m.profile_stats("w")[1][1:-1]
    return out


def work(case):
    """Every prognostic field read and written once per pass, and p written;
    the operations of the three substeps."""
    b = f = 0.
    for itot, jtot, ktot, _, _ in sizes(case):
        n = itot * jtot * ktot
        nf = 3 if case["kind"] == "channel" else 4
        b += (2 * nf + 1) * n * case["prec"] / 8
        per = 160. if case["kind"] == "channel" else 560.
        f += 3 * n * (per + 10. + 5. * (math.log2(itot) + math.log2(jtot))) * case.get("steps", 1)
        if case.get("monitored"):
            f += 40. * n
    return {"bytes": b, "flops": f}


# ---------------------------------------------------------------------------
# The same numbers in 64 bits, in plain torch
# ---------------------------------------------------------------------------
def X(a, n):
    return torch.roll(a, -n, 2)


def Y(a, n):
    return torch.roll(a, -n, 1)


def mid(a, b):
    return 0.5 * (a + b)


def sixth(v, a, b, c, d, e, f):
    """The 6th-order flux with 5th-order upwind dissipation."""
    return (v * (37. * (c + d) - 8. * (b + e) + (a + f)) / 60.
            - v.abs() * (10. * (d - c) - 5. * (e - b) + (f - a)) / 60.)


def fourth(v, a, b, c, d):
    return v * (7. * (b + c) - (a + d)) / 12. - v.abs() * (3. * (c - b) - (d - a)) / 12.


def low(a, v, sh):
    """The 6th-order flux through the low face along the axis of sh."""
    return sixth(v, sh(a, -3), sh(a, -2), sh(a, -1), a, sh(a, 1), sh(a, 2))


def koren(v, mm, m, p, pp):
    """The limited flux between m and p (Koren 1993)."""
    def face(up, upup, down):
        d = up - upup
        r = 2. * (down - up) / (torch.copysign(torch.ones_like(d), d) * d.abs().clamp_min(2.220446049250313e-16))
        return up + 0.5 * torch.minimum(r, ((1. + r) / 3.).clamp_max(2.)).clamp_min(0.) * d
    return torch.where(v >= 0, v * face(m, mm, p), v * face(p, pp, m))


class Exact:
    """The time step of one model in double."""

    def __init__(self, c, fields):
        self.c = c
        self.f = fields
        dev = fields["u"].device
        t = lambda a: torch.as_tensor(a, dtype=torch.float64, device=dev)[:, None, None]  # noqa: E731
        zc = np.asarray(c.z)
        z = np.concatenate([[-zc[0]], zc, [2. * c.zsize - zc[-1]]])
        zh = np.concatenate([[0.], 0.5 * (zc[:-1] + zc[1:]), [c.zsize]])
        self.z = zc
        self.dz = t(np.diff(zh))                     # ktot
        self.dzi = 1. / self.dz
        self.dzhi = 1. / t(np.diff(z))               # ktot + 1 half levels
        self.zh = zh
        self.dxi, self.dyi = c.itot / c.xsize, c.jtot / c.ysize
        self.t = {n: torch.zeros_like(a) for n, a in fields.items()}
        plane = torch.zeros_like(fields["u"][:1])
        self.zero = plane
        self.gradbot = plane.clone()                 # of theta, from the surface model
        self.mo = {n: plane.clone() for n in ("dudz", "dvdz", "dbdz")}
        self.dt, self.idt = c.dt, int(1e9 * c.dt + 0.5)
        self.p = None
        if c.surface:
            self.lut()
        if c.swbuffer:
            self.target = {n: fields[n].mean(dim=(1, 2), keepdim=True) for n in ("u", "v", "th")}

    # -- vertical neighbours --
    def padded(self, n):
        """Levels -1 .. ktot of u, v or theta."""
        a, c = self.f[n], self.c
        if n == "th":
            bot = a[:1] - self.gradbot / self.dzhi[:1]
            top = a[-1:] + c.stop / self.dzhi[-1:]
        else:
            bot = -a[:1]
            top = -a[-1:] if c.mbctop == mcases.BC_DIRICHLET else a[-1:]
        return torch.cat([bot, a, top])

    def zflux(self, a, v):
        """Advective flux through the half levels 0 .. ktot (v there)."""
        k = a.shape[0]
        out = torch.zeros_like(v)
        out[3:k - 2] = sixth(v[3:k - 2], a[:-5], a[1:-4], a[2:-3], a[3:-2], a[4:-1], a[5:])
        for q in (2, k - 2):
            out[q] = fourth(v[q], a[q - 2], a[q - 1], a[q], a[q + 1])
        for q in (1, k - 1):
            out[q] = v[q] * mid(a[q - 1], a[q])
        return out

    # -- surface layer --
    def functions(self, L):
        """The Monin-Obukhov flux factors and gradient functions."""
        zsl, z0m, z0h = float(self.z[0]), self.c.z0m, self.c.z0h

        def unstable(z, g):
            return (1. + g * z.abs() ** (2. / 3.)) ** -0.5

        def psi_u(phi):
            return 3. * torch.log((1. + 1. / phi) / 2.)

        def psim_s(z):
            return -2. / 3. * (z - 5. / 0.35) * torch.exp(-0.35 * z) - z - (10. / 3.) / 0.35

        def psih_s(z):
            return -2. / 3. * (z - 5. / 0.35) * torch.exp(-0.35 * z) - (1. + 2. / 3. * z) ** 1.5 - (10. / 3.) / 0.35 + 1.

        neg = L <= 0.
        z, zm, zt = zsl / L, z0m / L, z0h / L
        pos = lambda a: a.clamp_min(0.)  # noqa: E731
        pm = torch.where(neg, psi_u(unstable(z, 3.6)) - psi_u(unstable(zm, 3.6)), psim_s(pos(z)) - psim_s(pos(zm)))
        ph = torch.where(neg, psi_u(unstable(z, 7.9)) - psi_u(unstable(zt, 7.9)), psih_s(pos(z)) - psih_s(pos(zt)))
        fm = KAPPA / (math.log(zsl / z0m) - pm)
        fh = KAPPA / (math.log(zsl / z0h) - ph)
        return fm, fh, torch.where(neg, unstable(z, 3.6), 1. + 5. * z), torch.where(neg, unstable(z, 7.9), (1. + 4. * z) ** 2)

    def lut(self):
        """z/L against the Richardson number: 10000 entries, in float."""
        n = 10000
        dzl = (10. + 5.) / (9. * n / 10. - 1.)
        zt = np.zeros(n)
        zt[0] = -10.
        for q in range(1, 9 * n // 10):
            zt[q] = zt[q - 1] + dzl
        end, r, r0 = -(-1.e4 + 5.), 1.01, 1.e30
        while abs((r - r0) / r0) > 1.e-10:
            r0 = r
            r = (1. - (end / dzl) * (1. - r)) ** (1. / (n / 10.))
        for q in range(9 * n // 10, n):
            zt[q] = zt[q - 1] + dzl
            dzl *= r
        zl = (-zt[::-1]).astype(np.float32)
        dev = self.f["u"].device
        self.zl = torch.as_tensor(zl.copy(), device=dev)
        fm, _, _, _ = self.functions(float(self.z[0]) / self.zl.double())
        self.ri = (self.zl.double() * fm ** 3).to(torch.float32)

    def surface(self):
        c, f = self.c, self.f
        u, v, th = f["u"][:1], f["v"][:1], f["th"][:1]
        # Filtered wind speed at the cell centres.
        wx = lambda a: 0.5 * X(a, -1) + a + X(a, 1) + 0.5 * X(a, 2)  # noqa: E731
        wy = lambda a: 0.5 * Y(a, -1) + a + Y(a, 1) + 0.5 * Y(a, 2)  # noqa: E731
        uf = (Y(wx(u), -1) + wx(u) + Y(wx(u), 1)) / 9.
        vf = (X(wy(v), -1) + wy(v) + X(wy(v), 1)) / 9.
        du = (uf * uf + vf * vf).sqrt().clamp_min(0.1)
        zsl = float(self.z[0])
        ri = (-KAPPA * GRAV / THREF * c.sbot * zsl / du ** 3).to(torch.float32)
        n = torch.searchsorted(self.ri, ri.contiguous()).clamp(0, 9999)
        m = (n - 1).clamp_min(0)
        x0, x1, f0, f1 = self.zl[m], self.zl[n], self.ri[m], self.ri[n]
        zl = torch.where((n == 0) | (n == 9999), x1, x0 + (ri - f0) / (f1 - f0) * (x1 - x0)).double()
        fm, fh, phim, phih = self.functions(zsl / zl)
        us = du * fm
        c2 = us * fm
        self.uflux = -u * 0.5 * (X(c2, -1) + c2)
        self.vflux = -v * 0.5 * (Y(c2, -1) + c2)
        self.gradbot = -(c.sbot / (us * fh)) / zsl
        kz = KAPPA * zsl
        self.mo["dudz"] = mid(u, X(u, 1)) * fm / kz * phim
        self.mo["dvdz"] = mid(v, Y(v, 1)) * fm / kz * phim
        self.mo["dbdz"] = -(GRAV / THREF * c.sbot) / (kz * us) * phih

    # -- the terms --
    def viscosity(self):
        c, dxi, dyi = self.c, self.dxi, self.dyi
        u, v, w = self.f["u"], self.f["v"], torch.cat([self.f["w"], self.zero])
        th = self.padded("th")
        wt, wb = w[1:], w[:-1]
        xy = ((u - Y(u, -1)) * dyi + (v - X(v, -1)) * dxi) ** 2
        s2 = ((X(u, 1) - u) * dxi) ** 2 + ((Y(v, 1) - v) * dyi) ** 2 + ((wt - wb) * self.dzi) ** 2
        s2 += 0.125 * (xy + X(xy, 1) + Y(xy, 1) + X(Y(xy, 1), 1))
        up, vp = self.padded("u"), self.padded("v")
        xz = ((up[1:] - up[:-1]) * self.dzhi + (w - X(w, -1)) * dxi) ** 2
        yz = ((vp[1:] - vp[:-1]) * self.dzhi + (w - Y(w, -1)) * dyi) ** 2
        # At the surface the vertical gradients are the surface model's.
        wx, wy = ((w[:2] - X(w[:2], -1)) * dxi) ** 2, ((w[:2] - Y(w[:2], -1)) * dyi) ** 2
        s = 0.125 * (xz[1:] + X(xz[1:], 1) + xz[:-1] + X(xz[:-1], 1) + yz[1:] + Y(yz[1:], 1) + yz[:-1] + Y(yz[:-1], 1))
        s[0] = (0.5 * (self.mo["dudz"] ** 2 + self.mo["dvdz"] ** 2)
                + 0.125 * (wx + X(wx, 1) + wy + Y(wy, 1)).sum(dim=0, keepdim=True))[0]
        s2 = 2. * (s2 + s) + 1.e-9
        n2 = GRAV / THREF * 0.5 * (th[2:] - th[:-2]) * self.dzi
        n2[0] = self.mo["dbdz"][0]
        m0 = c.cs * (self.dz / (dxi * dyi)) ** (1. / 3.)
        zz = torch.as_tensor(self.z, dtype=torch.float64, device=u.device)[:, None, None]
        m2 = 1. / (1. / m0 ** 2 + 1. / (KAPPA * (zz + c.z0m)) ** 2)
        return m2 * s2.sqrt() * (1. - (n2 / s2 / c.tpr).clamp_max(1. - 1.e-9)).sqrt()

    def les(self, e):
        """Advection, Smagorinsky diffusion and buoyancy."""
        c, f, dxi, dyi = self.c, self.f, self.dxi, self.dyi
        u, v, s = f["u"], f["v"], f["th"]
        w = torch.cat([f["w"], self.zero])                           # half levels 0 .. ktot
        ep = torch.cat([e[:1], e, e[-1:]])
        eh = mid(ep[1:], ep[:-1])                                    # at the half levels
        up, vp = self.padded("u"), self.padded("v")
        txy = (mid(mid(e, X(e, -1)), Y(mid(e, X(e, -1)), -1)) + c.visc) * ((u - Y(u, -1)) * dyi + (v - X(v, -1)) * dxi)
        txz = (mid(eh, X(eh, -1)) + c.visc) * ((up[1:] - up[:-1]) * self.dzhi + (w - X(w, -1)) * dxi)
        tyz = (mid(eh, Y(eh, -1)) + c.visc) * ((vp[1:] - vp[:-1]) * self.dzhi + (w - Y(w, -1)) * dyi)

        def add(n, fx, fy, fz, zi):
            self.t[n][-fx.shape[0]:] += (X(fx, 1) - fx) * dxi + (Y(fy, 1) - fy) * dyi + (fz[1:] - fz[:-1]) * zi

        fz = txz.clone()
        fz[0], fz[-1] = -self.uflux[0], 0.
        add("u", 2. * (X(e, -1) + c.visc) * (u - X(u, -1)) * dxi - low(u, mid(u, X(u, -1)), X),
            txy - low(u, mid(v, X(v, -1)), Y), fz - self.zflux(u, mid(w, X(w, -1))), self.dzi)
        fz = tyz.clone()
        fz[0], fz[-1] = -self.vflux[0], 0.
        add("v", txy - low(v, mid(u, Y(u, -1)), X),
            2. * (Y(e, -1) + c.visc) * (v - Y(v, -1)) * dyi - low(v, mid(v, Y(v, -1)), Y),
            fz - self.zflux(v, mid(w, Y(w, -1))), self.dzi)
        # w at the half levels 1 .. ktot-1; its vertical fluxes at the full levels.
        wi = w[1:-1]
        vel = mid(w[:-1], w[1:])
        fz = torch.empty_like(vel)
        k = vel.shape[0]
        fz[2:-2] = sixth(vel[2:-2], w[:-5], w[1:-4], w[2:-3], w[3:-2], w[4:-1], w[5:])
        for q in (1, k - 2):
            fz[q] = fourth(vel[q], w[q - 1], w[q], w[q + 1], w[q + 2])
        for q in (0, k - 1):
            fz[q] = vel[q] * vel[q]
        fz = 2. * (e + c.visc) * (w[1:] - w[:-1]) * self.dzi - fz
        add("w", txz[1:-1] - low(wi, mid(u[1:], u[:-1]), X), tyz[1:-1] - low(wi, mid(v[1:], v[:-1]), Y),
            fz, self.dzhi[1:-1])
        self.t["w"][1:] += GRAV / THREF * (mid(s[1:], s[:-1]) - THREF)
        # theta
        tp = 1. / c.tpr
        if c.fluxlimit:
            ax, ay = koren(u, X(s, -2), X(s, -1), s, X(s, 1)), koren(v, Y(s, -2), Y(s, -1), s, Y(s, 1))
            az = torch.zeros_like(w)
            az[2:-2] = koren(w[2:-2], s[:-3], s[1:-2], s[2:-1], s[3:])
            # Upward through the lowest face and downward through the highest: unlimited.
            lim = koren(w[1], s[0], s[0], s[1], s[2])
            az[1] = torch.where(w[1] >= 0, w[1] * s[0], lim)
            lim = koren(w[-2], s[-3], s[-2], s[-1], s[-1])
            az[-2] = torch.where(w[-2] >= 0, lim, w[-2] * s[-1])
        else:
            ax, ay, az = low(s, u, X), low(s, v, Y), self.zflux(s, w)
        fz = torch.empty_like(w)
        fz[1:-1] = (eh[1:-1] * tp + c.svisc) * (s[1:] - s[:-1]) * self.dzhi[1:-1]
        fz[0], fz[-1] = -c.sbot, 0.
        add("th", (mid(e, X(e, -1)) * tp + c.svisc) * (s - X(s, -1)) * dxi - ax,
            (mid(e, Y(e, -1)) * tp + c.svisc) * (s - Y(s, -1)) * dyi - ay, fz - az, self.dzi)

    def buffer(self):
        c = self.c
        for n, z in (("u", self.z), ("v", self.z), ("th", self.z), ("w", self.zh[:-1])):
            sig = np.where(z >= c.buffer_zstart,
                           c.buffer_sigma * (np.maximum(z - c.buffer_zstart, 0.) / (c.zsize - c.buffer_zstart)) ** c.buffer_beta, 0.)
            sig = torch.as_tensor(sig, dtype=torch.float64, device=self.zero.device)[:, None, None]
            self.t[n] -= sig * (self.f[n] - (self.target[n] if n != "w" else 0.))

    def dns(self):
        """Advec_2, Diff_2 and the pressure force."""
        c, f, dxi, dyi = self.c, self.f, self.dxi, self.dyi
        u, v = f["u"], f["v"]
        w = torch.cat([f["w"], self.zero])
        up, vp = self.padded("u"), self.padded("v")

        def add(n, a, vx, vy, az, vz, zi, zhi):
            """Fluxes through the low faces; az: a with one more level on each side."""
            fx = c.visc * (a - X(a, -1)) * dxi - vx * mid(a, X(a, -1))
            fy = c.visc * (a - Y(a, -1)) * dyi - vy * mid(a, Y(a, -1))
            fz = c.visc * (az[1:] - az[:-1]) * zhi - vz * mid(az[1:], az[:-1])
            self.t[n][-a.shape[0]:] += (X(fx, 1) - fx) * dxi + (Y(fy, 1) - fy) * dyi + (fz[1:] - fz[:-1]) * zi

        add("u", u, mid(u, X(u, -1)), mid(v, X(v, -1)), up, mid(w, X(w, -1)), self.dzi, self.dzhi)
        add("v", v, mid(u, Y(u, -1)), mid(v, Y(v, -1)), vp, mid(w, Y(w, -1)), self.dzi, self.dzhi)
        add("w", w[1:-1], mid(u[1:], u[:-1]), mid(v[1:], v[:-1]), w, mid(w[1:], w[:-1]), self.dzhi[1:-1], self.dzi)
        self.t["u"] += -c.dpdx

    def pressure(self, sdt):
        c, f, t = self.c, self.f, self.t
        pu, pv, pw = (t[n] + f[n] / sdt for n in ("u", "v", "w"))
        pw = torch.cat([pw, self.zero])
        pw[0] = 0.
        rhs = (X(pu, 1) - pu) * self.dxi + (Y(pv, 1) - pv) * self.dyi + (pw[1:] - pw[:-1]) * self.dzi
        q = torch.fft.rfft2(rhs)
        dev = rhs.device
        lx = 2. * (torch.cos(2. * math.pi * torch.arange(q.shape[2], dtype=torch.float64, device=dev) / c.itot) - 1.) * self.dxi ** 2
        ly = 2. * (torch.cos(2. * math.pi * torch.arange(c.jtot, dtype=torch.float64, device=dev) / c.jtot) - 1.) * self.dyi ** 2
        lam = ly[:, None] + lx[None, :]
        dz, dzhi = self.dz[:, 0, 0], self.dzhi[:, 0, 0]
        k = c.ktot
        lo, hi = dz * dzhi[:-1], dz * dzhi[1:]
        den, work = [], []
        for n in range(k):
            b = dz[n] ** 2 * lam - (lo[n] + hi[n])
            if n == 0:
                b = b + lo[0]
            if n == k - 1:
                b = b + hi[n]
                b[0, 0] -= 2. * hi[n]
            r = dz[n] ** 2 * q[n]
            if n:
                m = lo[n] / den[-1]
                b = b - m * hi[n - 1]
                r = r - m * work[-1]
            den.append(b)
            work.append(r)
        q[k - 1] = work[-1] / den[-1]
        for n in range(k - 2, -1, -1):
            q[n] = (work[n] - hi[n] * q[n + 1]) / den[n]
        del den, work
        # The mean mode apart from the others: it is far larger than they are.
        mean = q[:, 0, 0].real.clone() / (c.itot * c.jtot)
        q[:, 0, 0] = 0.
        p = torch.fft.irfft2(q, s=(c.jtot, c.itot))
        t["u"] -= (p - X(p, -1)) * self.dxi
        t["v"] -= (p - Y(p, -1)) * self.dyi
        self.p = p + mean[:, None, None]
        t["w"][1:] -= (self.p[1:] - self.p[:-1]) * self.dzhi[1:-1]

    def cfl(self):
        f, c = self.f, self.c
        w = torch.cat([f["w"], self.zero])
        if c.advec == "2":
            s = mid(f["u"], X(f["u"], 1)).abs() * self.dxi + mid(f["v"], Y(f["v"], 1)).abs() * self.dyi
            return float((s + mid(w[1:], w[:-1]).abs() * self.dzi).max())
        one = torch.ones_like(f["u"])
        at = lambda a, sh: (37. * (a + sh(a, 1)) - 8. * (sh(a, -1) + sh(a, 2)) + sh(a, -2) + sh(a, 3)) / 60.  # noqa: E731
        wc = mid(w[1:], w[:-1])
        wc[1] = (7. * (w[1] + w[2]) - (w[0] + w[3])) / 12.
        wc[-2] = (7. * (w[-3] + w[-2]) - (w[-4] + w[-1])) / 12.
        wc[2:-2] = (37. * (w[2:-3] + w[3:-2]) - 8. * (w[1:-4] + w[4:-1]) + w[:-5] + w[5:]) / 60.
        return float(((at(f["u"], X).abs() * self.dxi + at(f["v"], Y).abs() * self.dyi) * one + wc.abs() * self.dzi).max())

    def step(self):
        c = self.c
        for q in range(3):
            e = self.viscosity() if c.diff == "smag2" else None
            if q == 0 and c.adaptivestep:
                dn = c.visc * float((self.dxi ** 2 + self.dyi ** 2 + self.dzi ** 2).max())
                self.idt = min(int(1e9 * 1e9 + 0.5), int(self.idt * c.cflmax / max(1.e-5, self.cfl() * self.dt)),
                               int(self.idt * c.dnmax / (self.dt * dn)))
                self.dt = self.idt / 1e9
            if c.surface:
                self.surface()
            if e is not None:
                self.les(e)
            else:
                self.dns()
            if c.swbuffer:
                self.buffer()
            self.pressure(CB[q] * self.dt)
            for n in self.f:
                self.f[n] = self.f[n] + CB[q] * self.dt * self.t[n]
                self.t[n] = self.t[n] * CA[(q + 1) % 3]


def exact(case, seed):
    outs = []
    for m, (itot, jtot, ktot, sbot, lapse) in enumerate(sizes(case)):
        c = setup(case, itot, jtot, ktot, sbot, lapse)
        ini = stored(case, initial(case, c, seed + 1000 * m))
        target = None
        if c.swbuffer:
            target = {n: a.mean(dim=(1, 2), keepdim=True) for n, a in initial(case, c, seed + 1000 * m).items()}
        off = THREF if case["prec"] == 32 else 0.
        x = Exact(c, {n: a.double() + (off if n == "th" else 0.) for n, a in ini.items()})
        if target:
            x.target = target
        for _ in range(case.get("steps", 1)):
            x.step()
        out = {n: a - off if n == "th" else a for n, a in x.f.items()}
        if case["kind"] == "les":
            out["p"] = x.p
        if case.get("monitored"):
            out["cfl"] = np.float64(x.cfl() * x.dt)
            for n in ("u", "v", "th", "w"):
                a = x.f[n]
                mean = a.mean(dim=(1, 2), keepdim=True)
                if n != "w":
                    out[n + "_mean"] = mean[:, 0, 0].cpu().numpy()
                out[n + "_var"] = ((a - mean) ** 2).mean(dim=(1, 2)).cpu().numpy()
        outs.append(out)
        del x
    return outs if case["kind"] == "ensemble" else outs[0]
