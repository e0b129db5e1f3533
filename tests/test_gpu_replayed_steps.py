"""Steps replayed as one graph launch against the same steps launched one by one
(timing on): the same kernels with the same arguments, so equal bit for bit."""
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


def run(mhh, case, precision, fused, replayed, steps):
    """Fields after `steps(model, run)`; launches counted."""
    m = mhh.Model(case, precision=precision)
    l0 = mhh.launch_count()
    mhh.Timing.enable(not replayed)
    try:
        steps(m, lambda n: m.run_steps(n, fused=fused))
        m.synchronize()
    finally:
        mhh.Timing.enable(False)
        mhh.Timing.reset()
    out = {n: m.get(n).copy() for n in case.prognostic_names()}
    launches = mhh.launch_count() - l0
    m.close()
    return out, launches


def plain(m, go):
    go(12)


def single(m, go):
    for _ in range(9):
        go(1)


def substeps(m, go):
    """Steps entered between substeps."""
    m.run_substeps(2, fused=True)
    go(5)
    m.run_substeps(1, fused=True)
    go(6)


def fields(m, go):
    """New values in the fields after the capture."""
    go(6)
    m.set("u", m.get("u")[..., ::-1].copy())
    go(3)


@pytest.mark.parametrize("steps", [plain, single, substeps, fields], ids=lambda f: f.__name__)
@pytest.mark.parametrize("fused", [True, False], ids=["fused", "modules"])
@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("kind", ["drycbl", "channel"])
def test_replayed(mhh, kind, precision, fused, steps):
    if kind == "drycbl":
        case = cases.drycbl(24, 20, 16, seed=81, dt=2.)
    else:
        case = cases.channel(24, 20, 16, seed=82, dt=2.e-4, adaptivestep=False)
    want, n0 = run(mhh, case, precision, fused, False, steps)
    got, n1 = run(mhh, case, precision, fused, True, steps)
    assert n0 == n1
    for n in want:
        assert np.array_equal(got[n], want[n]), n


def test_option_between(mhh):
    """An option set after the capture is honoured."""
    case = cases.drycbl(24, 20, 16, seed=83, dt=2.)

    def change(m, go):
        go(6)
        mhh.set_option("tendency_kernel", 0)
        mhh.set_option("tdma_kernel", 1)
        go(6)

    try:
        want, _ = run(mhh, case, 64, True, False, change)
        mhh.set_option("tendency_kernel", -1)
        mhh.set_option("tdma_kernel", -1)
        got, _ = run(mhh, case, 64, True, True, change)
    finally:
        mhh.set_option("tendency_kernel", -1)
        mhh.set_option("tdma_kernel", -1)
    for n in want:
        assert np.array_equal(got[n], want[n]), n


def test_streams_and_capture(mhh):
    """Another stream after the capture, and steps inside a caller's capture."""
    import torch
    case = cases.drycbl(24, 20, 16, seed=84, dt=2.)
    want, _ = run(mhh, case, 32, True, False, lambda m, go: go(12))
    m = mhh.Model(case, precision=32)
    m.run_steps(6)
    torch.cuda.synchronize()
    s = torch.cuda.Stream()
    m.set_stream(s.cuda_stream)
    m.run_steps(3)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        m.run_steps(1)
    with torch.cuda.stream(s):
        g.replay()
    m.run_steps(2)
    m.synchronize()
    for n in want:
        assert np.array_equal(m.get(n), want[n]), n
    m.set_stream(0)
    del g
    m.close()
