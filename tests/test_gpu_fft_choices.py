"""Choices of the float transforms that the other tests do not tell apart: 4 and
8 pairs of columns per tile at the one length that has the choice, and lengths
just outside the list that has stages of radix 8."""
import ctypes
import math

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


@pytest.mark.parametrize("itot,ktot", [(3, 6), (25, 7), (32, 10), (35, 6), (64, 13)])
def test_column_pairs(mhh, itot, ktot):
    """jtot = 32 in float: full and partial last tiles of 8 and of 16 columns,
    the same bits."""
    case = cases.drycbl(itot, 32, ktot, 100. * itot, 3200., 100. * ktot, seed=121, noise_z=400.)
    out = []
    for pairs in (4, 8):
        mhh.set_option("fft_column_pairs", pairs)
        try:
            m = mhh.Model(case, precision=32)
            m.run_steps(2)
            out.append({n: m.get(n) for n in case.prognostic_names() + ["p"]})
            m.close()
        finally:
            mhh.set_option("fft_column_pairs", 8)
    for n in out[0]:
        assert np.array_equal(out[0][n], out[1][n]), n


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("itot,jtot", [(1536, 5), (2048, 3), (6, 1536), (4, 2048), (3072, 2), (4096, 2), (80, 160)])
def test_lengths_without_radix_8(mhh, itot, jtot, precision):
    """Forward and back within 4 eps log2(itot jtot) of the largest coefficient,
    twice that after both."""
    import torch
    kern, _ = mhh.load()
    ktot = 3
    desc = mhh.GridDesc(itot, jtot, ktot, 1, 1, 1, 1.0, 1.0, 1.0)
    phys = mhh.Physics(visc=1e-5, svisc=1e-5, cs=0.23, tpr=1 / 3., dnmax=0.4, swmason=1, cflmax=1.,
                       thref0=300., thermo=0, surface=0, z0m=0.1, z0h=0.1)
    z = np.linspace(0.1, 0.9, ktot)
    h = ctypes.c_void_p()
    mhh.check(kern.mhh_ctx_create(ctypes.byref(desc), z.ctypes.data_as(ctypes.POINTER(ctypes.c_double)),
                                  precision, ctypes.byref(phys), ctypes.byref(h)))
    dt, eps = (torch.float64, 2.3e-16) if precision == 64 else (torch.float32, 6e-8)
    t = torch.from_numpy(np.random.default_rng(5).standard_normal((ktot, jtot, itot))).to("cuda", dt)
    x = t.double().cpu().numpy()

    def halfcomplex(a, axis):
        n = a.shape[axis]
        f = np.moveaxis(np.fft.fft(a, axis=axis), axis, 0)
        out = np.empty(f.shape)
        out[:n // 2 + 1] = f[:n // 2 + 1].real
        for k in range(1, (n + 1) // 2):
            out[n - k] = f[k].imag
        return np.moveaxis(out, 0, axis)

    tol = 4 * eps * math.log2(itot * jtot)
    mhh.check(kern.mhh_fft_forward(h, ctypes.c_void_p(t.data_ptr()), None))
    torch.cuda.synchronize()
    want = halfcomplex(halfcomplex(x, 2), 1)
    assert np.abs(t.double().cpu().numpy() - want).max() <= tol * np.abs(want).max()
    mhh.check(kern.mhh_fft_backward(h, ctypes.c_void_p(t.data_ptr()), None))
    torch.cuda.synchronize()
    assert np.abs(t.double().cpu().numpy() / (itot * jtot) - x).max() <= 2 * tol * np.abs(x).max()
    kern.mhh_ctx_destroy(h)
