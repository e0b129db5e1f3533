"""The DNS tendencies in flux form (mhh_tend_2.cu: Advec_2 + Diff_2, every face
flux once) against the per-cell kernel, at the edges of its 32 x 8 tiles and of
its level chunks, with and without the scalar, buoyancy and the pressure force."""
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


def make(itot, jtot, ktot, thermo):
    c = cases.channel(itot, jtot, ktot, seed=71, dt=2.e-4, adaptivestep=False)
    if thermo:
        c.thermo, c.svisc, c.swlspres = True, 1. / 130., False
        c.sbcbot, c.sbctop, c.sbot, c.stop = cases.BC_DIRICHLET, cases.BC_NEUMANN, 301., 0.2
        rng = np.random.default_rng(72)
        c.fields["th"] = 300. + 0.1 * rng.standard_normal((ktot, jtot, itot))
    return c


@pytest.mark.parametrize("thermo", [False, True], ids=["channel", "thermo"])
@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("itot,jtot,ktot", [(4, 3, 2), (30, 7, 9), (32, 8, 8), (35, 9, 65), (64, 16, 129), (98, 25, 66)])
def test_flux_form_against_per_cell(mhh, itot, jtot, ktot, precision, thermo):
    """One substep in both forms, which round the same sums in another order.
    FP64: 1e-12, the bound of the channel against the oracle.  Float: the flux
    form is no further from FP64 than the per-cell form (half as much again for
    two samples of the same round-off, which the pressure solve amplifies: on
    the tallest grid here either form is 4e-6 from FP64 in w)."""
    case = make(itot, jtot, ktot, thermo)

    def step(variant, prec):
        mhh.set_option("tendency_kernel", variant)
        try:
            m = mhh.Model(case, precision=prec)
            m.run_substeps(1, fused=True)
            out = {n: case.interior(m.get(n)) - (300. if n == "th" else 0.) for n in case.prognostic_names()}
            m.close()
        finally:
            mhh.set_option("tendency_kernel", -1)
        return out

    flux, cell = step(2, precision), step(0, precision)
    exact = step(0, 64)
    for n, a in flux.items():
        norm = np.linalg.norm(exact[n])
        assert np.isfinite(a).all()
        if precision == 64:
            assert np.linalg.norm(a - cell[n]) <= 1e-12 * norm, n
        else:
            ef, ec = np.linalg.norm(a - exact[n]) / norm, np.linalg.norm(cell[n] - exact[n]) / norm
            print(n, ef, ec)
            assert ef <= 1.5 * ec + 1e-7, (n, ef, ec)
