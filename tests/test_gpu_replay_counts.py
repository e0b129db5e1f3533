"""Which steps are replayed as one graph launch, and that a change after the
capture is honoured: the same steps launched one by one (timing on) give the
same bits."""
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


def buffered():
    case = cases.drycbl(24, 20, 16, seed=98, dt=2.)
    rng = np.random.default_rng(99)
    for n in ("u", "v"):
        case.fields[n] = rng.normal(1., 0.3, (16, 20, 24))
    case.swbuffer, case.buffer_zstart, case.buffer_sigma = True, 2500., 0.01
    return case


@pytest.mark.parametrize("fused", [True, False], ids=["fused", "modules"])
def test_replayed_count(mhh, fused):
    m = mhh.Model(cases.drycbl(24, 20, 16, seed=98, dt=2.), precision=32)
    m.run_steps(3, fused=fused)
    assert m.replayed_steps() == 0
    m.run_steps(9, fused=fused)
    assert m.replayed_steps() == 9
    mhh.Timing.enable(True)
    m.run_steps(2, fused=fused)
    m.synchronize()
    mhh.Timing.enable(False)
    mhh.Timing.reset()
    assert m.replayed_steps() == 9
    m.run_steps(1, fused=fused)
    assert m.replayed_steps() == 10
    m.run_steps(4, fused=not fused)         # other launches: three one by one again
    assert m.replayed_steps() == 11
    m.close()


def test_adaptive_is_not_replayed(mhh):
    m = mhh.Model(cases.channel(24, 20, 16, seed=98, dt=2.e-4, adaptivestep=True), precision=64)
    m.run_steps(6)
    assert m.replayed_steps() == 0
    m.close()


def profile(mhh, m, tmp):
    m.set_buffer_profile("u", np.full(m.grid.kcells, 3.))


def limiter(mhh, m, tmp):
    kern, _ = mhh.load()
    mhh.check(kern.mhh_advec_2i5_set_fluxlimit(m.ctx(), 1), "fluxlimit")


def option(mhh, m, tmp):
    kern, _ = mhh.load()
    for n, v in ((b"tendency_kernel", 0), (b"tdma_kernel", 1), (b"viscosity_kchunk", 4)):
        mhh.check(kern.mhh_ctx_set_option(m.ctx(), n, v), "option")


def layer(mhh, m, tmp):
    kern, _ = mhh.load()
    mhh.check(kern.mhh_buffer_setup(m.ctx(), 1000., 0.02, 1.), "buffer")


def time_step(mhh, m, tmp):
    """A restart of another step: its time step holds from then on."""
    case = buffered()
    case.dt = 1.
    other = mhh.Model(case, precision=m.precision)
    other.run_steps(2)
    t = other.save(str(tmp))
    other.close()
    m.load(str(tmp), t)
    assert m.dt() == 1.


@pytest.mark.parametrize("change", [profile, limiter, option, layer, time_step], ids=lambda f: f.__name__)
@pytest.mark.parametrize("fused", [True, False], ids=["fused", "modules"])
@pytest.mark.parametrize("precision", [64, 32])
def test_change_after_capture(mhh, tmp_path, precision, fused, change):
    case = buffered()
    out = []
    for replayed in (False, True):
        m = mhh.Model(case, precision=precision)
        tmp = tmp_path / str(replayed)
        tmp.mkdir()
        mhh.Timing.enable(not replayed)
        try:
            m.run_steps(6, fused=fused)
            assert m.replayed_steps() == (3 if replayed else 0)
            change(mhh, m, tmp)
            m.run_steps(6, fused=fused)
            m.synchronize()
            assert m.replayed_steps() == (6 if replayed else 0)
        finally:
            mhh.Timing.enable(False)
            mhh.Timing.reset()
        out.append({n: m.get(n).copy() for n in case.prognostic_names()})
        m.close()
    for n in out[0]:
        assert np.array_equal(out[0][n], out[1][n]), n


def test_two_threads(mhh):
    """Two models stepped by two threads, captured while the other launches."""
    import threading
    made = [cases.drycbl(24, 20, 16, seed=100 + q, dt=2.) for q in range(2)]
    want = []
    for c in made:
        m = mhh.Model(c, precision=32)
        m.run_steps(40)
        want.append({n: m.get(n).copy() for n in c.prognostic_names()})
        m.close()
    import torch
    models = [mhh.Model(c, precision=32) for c in made]
    streams = [torch.cuda.Stream() for _ in models]
    fails = []

    def steps(m, s):
        try:
            m.set_stream(s.cuda_stream)
            for _ in range(40):
                m.run_steps(1)
            m.synchronize()
        except Exception as e:
            fails.append(e)

    ts = [threading.Thread(target=steps, args=a) for a in zip(models, streams)]
    n0 = mhh.launch_count()
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not fails, fails
    launched = mhh.launch_count() - n0
    for m, w in zip(models, want):
        assert m.replayed_steps() == 37
        for n in w:
            assert np.array_equal(m.get(n), w[n]), n
        m.set_stream(0)
        m.close()
    # As many kernels as the same steps one by one.
    m = mhh.Model(made[0], precision=32)
    mhh.Timing.enable(True)
    n0 = mhh.launch_count()
    m.run_steps(40)
    m.synchronize()
    mhh.Timing.enable(False)
    mhh.Timing.reset()
    assert launched == 2 * (mhh.launch_count() - n0)
    m.close()
