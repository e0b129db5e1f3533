"""The column-resident tridiagonal solves (mhh_pres.cu) against the sweeps
through global memory, at the heights where the number of column groups per
block changes, on odd and even sides, and above the tallest column that fits
in shared memory."""
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
    mhh.set_option("tdma_kernel", variant)
    try:
        m = mhh.Model(case, precision=precision)
        m.run_substeps(1, fused=True)
        out = case.interior(m.get("p"))
        m.close()
    finally:
        mhh.set_option("tdma_kernel", -1)
    return out


SIZES = [(12, 10, 6), (15, 9, 7), (9, 14, 65), (64, 48, 129), (35, 21, 258), (8, 6, 520), (5, 7, 1030),
         (6, 5, 2100), (4, 3, 4200), (3, 4, 8300)]


@pytest.mark.parametrize("itot,jtot,ktot", SIZES)
@pytest.mark.parametrize("precision", [64, 32])
def test_resident_columns(mhh, itot, jtot, ktot, precision):
    """The solution p.  FP64: the reference-order solve against the rescaled
    recurrence; the 1-D mean-mode problem has a condition number of about
    ktot^2, so the two orders of rounding differ by a few eps ktot^2.  FP32:
    the mixed solve against FP64 sweeps of every group, at the bound of the
    mixed solve, 2e-6 (the velocities of a flow at rest are differences of p
    far below its float rounding, so they say nothing here)."""
    case = cases.drycbl(itot, jtot, ktot, 100. * itot, 100. * jtot, 4000., seed=61, noise_z=1000.)
    a, b = solve(mhh, case, precision, -1), solve(mhh, case, precision, 1)
    eps = 2.2e-16
    assert np.isfinite(a).all()
    err = np.linalg.norm(a - b) / np.linalg.norm(b)
    assert err <= (8 * eps * ktot**2 + 1e-13 if precision == 64 else 2e-6), err
