"""Device memory of a context and its estimate, by which served jobs are
admitted."""
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


@pytest.mark.parametrize("itot,jtot,ktot", [(256, 256, 256), (512, 256, 90), (64, 48, 3300), (48, 40, 4500)])
@pytest.mark.parametrize("levels", ["uniform", "stretched"])
@pytest.mark.parametrize("precision", [64, 32])
def test_context_bytes(mhh, itot, jtot, ktot, precision, levels):
    """The packed field and the work array, 52 bytes per column group and level
    for the elimination tables (in FP32 contexts up to 16 more, for the groups
    that sweep in FP64) and 48 MB of everything else and allocation granularity;
    and no more than the estimate, which exceeds it by at most 100 MB and those
    tables."""
    from microhh_gb300 import cases
    kern, _ = mhh.load()
    # Cells 100 m wide and 40 m high, whose sweeps all damp but the mean's, or
    # 2 m of stretched levels, where none does.
    zsize = 2. if levels == "stretched" else 40. * ktot
    desc = mhh.GridDesc(itot, jtot, ktot, 3, 3, 1, 100. * itot, 100. * jtot, zsize)
    phys = mhh.Physics(visc=1e-5, svisc=1e-5, cs=0.23, tpr=1 / 3., dnmax=0.4, swmason=1, cflmax=1.,
                       thref0=300., thermo=1, surface=1, z0m=0.1, z0h=0.1)
    z = np.ascontiguousarray(cases.stretched_channel_z(ktot) if levels == "stretched" else cases.uniform_z(ktot, zsize))
    h, got, est = ctypes.c_void_p(), ctypes.c_size_t(), ctypes.c_size_t()
    kern.mhh_ctx_estimate_bytes.argtypes = [ctypes.POINTER(mhh.GridDesc), ctypes.c_int, ctypes.POINTER(ctypes.c_size_t)]
    mhh.check(kern.mhh_ctx_estimate_bytes(ctypes.byref(desc), precision, ctypes.byref(est)))
    mhh.check(kern.mhh_ctx_create(ctypes.byref(desc), z.ctypes.data_as(ctypes.POINTER(ctypes.c_double)),
                                  precision, ctypes.byref(phys), ctypes.byref(h)))
    mhh.check(kern.mhh_ctx_device_bytes(h, ctypes.byref(got)))
    kern.mhh_ctx_destroy(h)
    groups = (itot // 2 + 1) * (jtot // 2 + 1) * ktot
    want = itot * jtot * ktot * (precision // 8 + 8) + 52 * groups + 48e6
    listed = 16 * groups if precision == 32 else 0
    assert got.value <= want + (listed if levels == "stretched" else 0), (got.value / 1e6, want / 1e6)
    assert got.value <= est.value <= want + listed + 100e6, (got.value / 1e6, est.value / 1e6, want / 1e6)
