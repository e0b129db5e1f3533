"""The tallest columns that the column-resident solves keep in shared memory
(mhh_tdma.cu: 4411 levels in the mixed solve of the FP32 form, 3185 in FP64) and
the next height, which sweeps through global memory."""
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


def solve(mhh, case, precision, variant):
    """p of random velocities whose w has no mean at any level (the mean mode's
    p would hide the other modes below its rounding)."""
    kern, _ = mhh.load()
    rng = np.random.default_rng(132)
    m = mhh.Model(case, precision=precision)
    for n in ("u", "v", "w"):
        a = rng.standard_normal((case.ktot, case.jtot, case.itot))
        if n == "w":
            a -= a.mean(axis=(1, 2), keepdims=True)
            a[0] = 0.
        m.set(n, case.embed(a))
    f, b = m.device_fields()
    mhh.check(kern.mhh_ctx_set_option(m.ctx(), b"tdma_kernel", variant), "option")
    for p in (f.u, f.v, f.w):
        mhh.check(kern.mhh_boundary_cyclic(m.ctx(), p, 3, None), "cyclic")
    mhh.check(kern.mhh_pres_2_exec(m.ctx(), ctypes.byref(f), 1., None), "pres_2")
    m.synchronize()
    out = case.interior(m.get("p"))
    m.close()
    return out


@pytest.mark.parametrize("itot,jtot", [(6, 5), (3, 4)])
@pytest.mark.parametrize("precision,ktot", [(32, 4411), (32, 4412), (64, 3185), (64, 3186)])
def test_tallest_columns(mhh, itot, jtot, ktot, precision):
    """p against the other solves: in FP64 within a few eps ktot^2 (the condition
    number of the mean mode), in FP32 within the bound of the mixed solve, 2e-6.
    Cells 40 m high and 100 m wide, whose columns damp and so sweep in float in
    the mixed solve: its bits differ from the FP64 sweeps', which the height
    above takes."""
    case = cases.drycbl(itot, jtot, ktot, 100. * itot, 100. * jtot, 40. * ktot, seed=131, noise_z=4000.)
    auto = solve(mhh, case, precision, -1)
    assert np.isfinite(auto).all()
    for variant in (0, 1, 2):
        other = solve(mhh, case, precision, variant)
        err = np.linalg.norm(auto - other) / np.linalg.norm(other)
        assert err <= (8 * 2.2e-16 * ktot**2 + 1e-13 if precision == 64 else 2e-6), (variant, err)
        if precision == 32 and variant == 1:
            assert np.array_equal(auto, other) == (ktot > 4411)
