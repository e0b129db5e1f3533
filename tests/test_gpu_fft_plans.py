"""The run-time-plan transforms (every length but 32 in float; stages of radix
2 to 12) against numpy's DFT in halfcomplex order and back."""
import ctypes
import math

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


def halfcomplex(a, axis):
    n = a.shape[axis]
    f = np.moveaxis(np.fft.fft(a, axis=axis), axis, 0)
    out = np.empty(f.shape)
    out[:n // 2 + 1] = f[:n // 2 + 1].real
    for k in range(1, (n + 1) // 2):
        out[n - k] = f[k].imag
    return np.moveaxis(out, 0, axis)


# Every radix alone, its products, odd and even sides, the longest plans, and a
# length whose tile holds fewer than eight pairs.
SIZES = [(2, 3), (4, 5), (6, 7), (8, 9), (10, 14), (15, 12), (18, 21), (25, 20), (27, 28), (35, 30), (49, 45), (54, 81),
         (63, 100), (75, 105), (90, 125), (150, 189), (243, 6), (250, 343), (486, 7), (5, 490), (720, 3), (1000, 4),
         (3, 2187), (2100, 2)]


@pytest.mark.parametrize("offset", [0, 1], ids=["aligned", "offset"])
@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("itot,jtot", SIZES)
def test_plan(mhh, itot, jtot, precision, offset):
    """Within 4 eps log2(itot jtot) of the largest coefficient (a transform's
    error grows with the square root of its stages; 4 allows the worst point),
    with the data aligned and one element past an aligned address."""
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
    dt = torch.float64 if precision == 64 else torch.float32
    eps = 2.3e-16 if precision == 64 else 6e-8
    x = np.random.default_rng(5).standard_normal((ktot, jtot, itot))
    buf = torch.empty(x.size + offset, dtype=dt, device="cuda")
    t = buf[offset:].view(ktot, jtot, itot)
    t.copy_(torch.from_numpy(x))
    x = t.double().cpu().numpy()
    tol = 4 * eps * math.log2(itot * jtot)
    mhh.check(kern.mhh_fft_forward(h, ctypes.c_void_p(t.data_ptr()), None))
    torch.cuda.synchronize()
    want = halfcomplex(halfcomplex(x, 2), 1)
    assert np.abs(t.double().cpu().numpy() - want).max() <= tol * np.abs(want).max()
    mhh.check(kern.mhh_fft_backward(h, ctypes.c_void_p(t.data_ptr()), None))
    torch.cuda.synchronize()
    n = itot * jtot
    assert np.abs(t.double().cpu().numpy() / n - x).max() <= 2 * tol * np.abs(x).max()
    kern.mhh_ctx_destroy(h)


# The lengths of radix 8: 2^a, 2^a 3, and 128, 256 and 512 in frequency.
EIGHTS = [(16, 48), (64, 96), (128, 192), (256, 384), (512, 128), (768, 256), (1024, 512)]


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("itot,jtot", EIGHTS)
def test_eights(mhh, itot, jtot, precision):
    test_plan(mhh, itot, jtot, precision, 0)
