"""Infinities in the pressure solve stay where the arithmetic puts them."""
import ctypes

import numpy as np
import pytest

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


@pytest.mark.parametrize("axis", ["x", "y", "xy"])
@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("n", [2, 3, 5, 7, 8, 10, 14, 20, 32, 48, 64, 96, 150])
def test_inverse_mean(mhh, n, precision, axis):
    """The inverse transform of rows that are finite beside rows with an
    infinite mean, which are transformed in pairs: a finite row's values are
    those without its partner, the other's are infinite.  Columns of the xy
    case are adjacent pairs, whose sums and differences are infinite and not
    NaN."""
    import torch
    kern, _ = mhh.load()
    itot, jtot = {"x": (n, 1), "y": (1, n), "xy": (2, n)}[axis]
    h = context(mhh, itot, jtot, 4, precision)
    t = torch.rand((4, jtot, itot), dtype=torch.float64 if precision == 64 else torch.float32, device="cuda")
    plain = t.clone()
    if axis == "xy":
        t[:, 0, 1] = float("inf")
    else:
        t[1, 0, 0] = t[2, 0, 0] = float("inf")
    for a in (plain, t):
        mhh.check(kern.mhh_fft_backward(h, ctypes.c_void_p(a.data_ptr()), None))
    torch.cuda.synchronize()
    kern.mhh_ctx_destroy(h)
    if axis == "xy":
        assert bool(torch.isinf(t).all())
    else:
        assert torch.equal(t[0], plain[0]) and torch.equal(t[3], plain[3])
        assert bool(torch.isinf(t[1]).all()) and bool(torch.isinf(t[2]).all())


@pytest.mark.parametrize("ktot", [3, 8, 301, 3300])
@pytest.mark.parametrize("level", ["bottom", "top"])
def test_column_quotients(mhh, ktot, level):
    """FP64, the reference's order of operations on one column: an infinite
    right-hand side at its bottom or top level gives the quotients x/d, signed
    infinities, as in the recurrence written out here."""
    from microhh_gb300 import cases
    kern, _ = mhh.load()
    case = cases.channel(1, 1, ktot, seed=95, dt=1.e-4, adaptivestep=False)
    m = mhh.Model(case, precision=64)
    w = m.get("w")
    # w at the lower face of the lowest cell, or at the upper of the highest.
    w[1 if level == "bottom" else ktot + 1] = np.inf
    m.set("w", w)
    f, _ = m.device_fields()
    mhh.check(kern.mhh_pres_2_exec(m.ctx(), ctypes.byref(f), 1.e-4, None), "pres_2")
    m.synchronize()
    got = case.interior(m.get("p")).ravel()
    dz, dzhi = m.profile("dz")[1:-1], m.profile("dzhi")[1:]
    m.close()
    a, c = dz * dzhi[:-1], dz * dzhi[1:]
    rhs = np.zeros(ktot)
    rhs[0 if level == "bottom" else -1] = -np.inf if level == "bottom" else np.inf
    b = -(a + c)
    b[0] += a[0]
    b[-1] -= c[-1]
    y, den = np.zeros(ktot), np.zeros(ktot)
    den[0] = b[0]
    y[0] = rhs[0] / den[0]
    for k in range(1, ktot):
        den[k] = b[k] - a[k] * (c[k - 1] / den[k - 1])
        y[k] = (rhs[k] - a[k] * y[k - 1]) / den[k]
    for k in range(ktot - 2, -1, -1):
        y[k] -= c[k] / den[k] * y[k + 1]
    assert np.array_equal(np.sign(got), np.sign(y)) and np.isinf(got).all()
