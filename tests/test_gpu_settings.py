"""The number of a context's settings (mhh_ctx_settings), by which a driver that
keeps captured launches learns that one changed."""
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


@pytest.fixture()
def ctx(mhh):
    kern, _ = mhh.load()
    kern.mhh_ctx_settings.restype = ctypes.c_ulonglong
    kern.mhh_ctx_settings.argtypes = [ctypes.c_void_p]
    m = mhh.Model(cases.drycbl(12, 10, 6, seed=96), precision=64)
    yield kern, m.ctx()
    m.close()


# Every accepted change, and the same refused.
CHANGES = [("option", ("tendency_kernel", 0), ("tendency_kernel", 3)), ("option", ("viscosity_kernel", 0), ("viscosity_kernel", 2)),
           ("option", ("tdma_kernel", 1), ("tdma_kernel", 4)), ("option", ("pres_fuse", 0), ("pres_fuse", 2)),
           ("option", ("fft_column_pairs", 4), ("fft_column_pairs", 5)), ("option", ("tendency_kchunk", 8), ("tendency_kchunk", 7)),
           ("ctx", ("tendency_kernel", 0), ("tendency_kernel", 3)), ("ctx", ("tdma_kernel", 1), ("tdma_kernel", 4)),
           ("ctx", ("viscosity_kchunk", 16), ("unknown", 1)), ("limit", (1,), None), ("surface", (2,), (7,)),
           ("buffer", (0.5, 2., 2.), None), ("profile", ("u",), ("q",))]
DEFAULTS = [("tendency_kernel", -1), ("viscosity_kernel", -1), ("tdma_kernel", -1), ("pres_fuse", 1), ("fft_column_pairs", 8),
            ("tendency_kchunk", 0)]


@pytest.mark.parametrize("kind,good,bad", CHANGES, ids=lambda v: "-".join(map(str, v)) if isinstance(v, tuple) else str(v))
def test_settings_number(mhh, ctx, kind, good, bad):
    """It stays after a refused change and grows with an accepted one."""
    kern, c = ctx
    prof = np.zeros(64)
    dp = prof.ctypes.data_as(ctypes.POINTER(ctypes.c_double))
    call = {"option": lambda n, v: kern.mhh_set_option(n.encode(), v),
            "ctx": lambda n, v: kern.mhh_ctx_set_option(c, n.encode(), v),
            "limit": lambda v: kern.mhh_advec_2i5_set_fluxlimit(c, v),
            "surface": lambda v: kern.mhh_boundary_surface_init(c, v),
            "buffer": lambda *v: kern.mhh_buffer_setup(c, *v),
            "profile": lambda n: kern.mhh_buffer_set_profile(c, n.encode(), dp)}[kind]
    if kind == "profile":
        assert kern.mhh_buffer_setup(c, 0.5, 2., 2.) == 0
    try:
        n0 = kern.mhh_ctx_settings(c)
        if bad is not None:
            assert call(*bad) != 0
            assert kern.mhh_ctx_settings(c) == n0
        assert call(*good) == 0
        assert kern.mhh_ctx_settings(c) > n0
    finally:
        if kind == "option":
            for n, v in DEFAULTS:
                kern.mhh_set_option(n.encode(), v)
