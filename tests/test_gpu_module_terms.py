"""Advec_2i5 and Diff_smag2 alone (the module-by-module step) in flux form against
the per-cell kernel, at the edges of the 32 x 8 tiles and of the level chunks, with
the surface model, without it and without the scalar, and with the flux limiter."""
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


def make(itot, jtot, ktot, kind):
    c = cases.drycbl(itot, jtot, ktot, seed=73, dt=1.)
    rng = np.random.default_rng(74)
    for n, s in (("u", 1.), ("v", 1.), ("w", 0.3), ("th", 0.2)):
        a = s * rng.standard_normal((ktot, jtot, itot))
        if n == "w":
            a[0] = 0.
        c.fields[n] = a + (c.fields[n] if n == "th" else 0.)
    if kind == "limited":
        c.fluxlimit = True
    if kind == "neutral":
        c.thermo = c.surface = False
        del c.fields["th"]
    if kind == "noslip":
        c.surface = False
    return c


@pytest.mark.parametrize("kind", ["surface", "limited", "neutral", "noslip"])
@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("itot,jtot,ktot", [(6, 5, 6), (30, 7, 9), (32, 8, 8), (35, 9, 65), (64, 16, 67)])
def test_flux_form_against_per_cell(mhh, itot, jtot, ktot, precision, kind):
    """One substep.  FP64: 1e-12, the bound of the two forms of the whole
    tendency.  Float: no further from FP64 than the per-cell form (half as much
    again for two samples of the same round-off)."""
    case = make(itot, jtot, ktot, kind)

    def step(variant, prec):
        mhh.set_option("tendency_kernel", variant)
        try:
            m = mhh.Model(case, precision=prec)
            m.run_substeps(1, fused=False)
            out = {n: case.interior(m.get(n)) - (300. if n == "th" else 0.) for n in case.prognostic_names()}
            m.close()
        finally:
            mhh.set_option("tendency_kernel", -1)
        return out

    flux, cell, exact = step(2, precision), step(0, precision), step(0, 64)
    for n, a in flux.items():
        norm = np.linalg.norm(exact[n])
        assert np.isfinite(a).all()
        if precision == 64:
            assert np.linalg.norm(a - cell[n]) <= 1e-12 * norm, n
        else:
            ef, ec = np.linalg.norm(a - exact[n]) / norm, np.linalg.norm(cell[n] - exact[n]) / norm
            assert ef <= 1.5 * ec + 1e-7, (n, ef, ec)
