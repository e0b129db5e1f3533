"""Grids whose levels reach the number of blocks that a launch may have along y
and z (65535)."""
import ctypes

import numpy as np
import pytest

from microhh_gb300 import cases

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def mhh():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import microhh_gb300
    microhh_gb300.load()
    return microhh_gb300


def context(mhh, itot, jtot, ktot, precision):
    kern, _ = mhh.load()
    desc = mhh.GridDesc(itot, jtot, ktot, 1, 1, 1, 1.0, 1.0, 1.0)
    phys = mhh.Physics(visc=1e-5, svisc=1e-5, cs=0.23, tpr=1 / 3., dnmax=0.4, swmason=1, cflmax=1.,
                       thref0=300., thermo=0, surface=0, z0m=0.1, z0h=0.1)
    z = (np.arange(ktot) + 0.5) / ktot
    h = ctypes.c_void_p()
    mhh.check(kern.mhh_ctx_create(ctypes.byref(desc), z.ctypes.data_as(ctypes.POINTER(ctypes.c_double)),
                                  precision, ctypes.byref(phys), ctypes.byref(h)))
    return h


@pytest.mark.parametrize("ktot", [65533, 65534, 70000])
@pytest.mark.parametrize("precision", [64, 32])
def test_rk3_levels(mhh, ktot, precision):
    """a + cB dt at and cA at (zero everywhere after the last substep): three
    roundings of a sum of order one in the fields' precision."""
    import torch
    kern, _ = mhh.load()
    itot, jtot, dt = 4, 3, 0.7
    h = context(mhh, itot, jtot, ktot, precision)
    tt = torch.float64 if precision == 64 else torch.float32
    tol = 4 * (2.3e-16 if precision == 64 else 6e-8)
    rng = np.random.default_rng(91)
    shape = (ktot + 2, jtot + 2, itot + 2)
    inside = (slice(1, -1),) * 3
    for substep in (0, 2):
        a = torch.tensor(rng.standard_normal(shape), dtype=tt, device="cuda")
        at = torch.tensor(rng.standard_normal(shape), dtype=tt, device="cuda")
        a0, t0 = a.double().cpu().numpy(), at.double().cpu().numpy()
        mhh.check(kern.mhh_timeloop_rk3(h, a.data_ptr(), at.data_ptr(), substep, dt, None), "rk3")
        torch.cuda.synchronize()
        want, wt = a0.copy(), t0.copy()
        want[inside] += (1. / 3., 15. / 16., 8. / 15.)[substep] * dt * t0[inside]
        if substep == 2:
            wt[:] = 0.
        else:
            wt[inside] *= -5. / 9.
        scale = np.abs(a0).max() + np.abs(t0).max()
        assert np.abs(a.double().cpu().numpy() - want).max() <= tol * scale
        assert np.abs(at.double().cpu().numpy() - wt).max() <= tol * scale
    kern.mhh_ctx_destroy(h)


@pytest.mark.parametrize("ktot", [65500, 65533])
@pytest.mark.parametrize("precision", [64, 32])
def test_ghosts_of_the_tallest_grids(mhh, ktot, precision):
    """The ghost cells at the start of a substep: periodic images, and the
    no-slip wall levels minus the lowest and highest cell, to the last bit."""
    kern, _ = mhh.load()
    case = cases.channel(5, 4, ktot, seed=92, dt=1.e-9, adaptivestep=False)
    m = mhh.Model(case, precision=precision)
    f, b = m.device_fields()
    cfg = mhh.SubstepConfig(advec=mhh.ADVEC_2, diff=mhh.DIFF_2, swlspres=1, dpdx=-1., mbcbot=0, mbctop=0, sbcbot=2, sbctop=2)
    mhh.check(kern.mhh_substep_begin(m.ctx(), ctypes.byref(cfg), ctypes.byref(f), ctypes.byref(b), None), "substep_begin")
    m.synchronize()
    for n in ("u", "v", "w"):
        got = m.get(n)
        inner = got[1:-1, 1:-1, 1:-1]
        want = np.pad(inner, ((0, 0), (1, 1), (1, 1)), mode="wrap")
        assert np.array_equal(got[1:-1], want), n
        if n != "w":
            assert np.array_equal(got[0], -want[0]) and np.array_equal(got[-1], -want[-1]), n
    m.close()
