"""The ensemble's autotuner compares its choices with what a context does by
itself."""
import re

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


def test_choices_include_the_automatic_one(mhh):
    """The time of the choice beside the automatic one's, which it may not exceed
    but for the noise of two steps."""
    grids = [(32, 32, 32), (64, 48, 40), (128, 128, 96)]
    models = [mhh.Model(cases.drycbl(*g, seed=141), precision=mhh.FP32) for g in grids]
    ens = mhh.Ensemble(models)
    report = ens.autotune()
    ens.close()
    for m in models:
        m.close()
    for g in grids:
        r = re.search(r"%dx%dx%d: tendency (-?\d+)/(-?\d+) viscosity (-?\d+)/(-?\d+) \(([\d.]+) ms/step, automatic ([\d.]+)\)" % g, report)
        assert r, report
        # Both or neither of a kernel's variant and height are the context's own.
        assert (r[1] == "-2") == (r[2] == "-2") and (r[3] == "-2") == (r[4] == "-2"), report
        assert float(r[5]) <= 1.25 * float(r[6]), report
