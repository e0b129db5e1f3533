"""A setting or a time step changed between two calls of an ensemble that
replays captured launches holds from the next step on: the same bits as the
members' own launches (streams mode)."""
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


def made():
    out = []
    for q, (i, j, k) in enumerate([(24, 20, 16), (24, 20, 16), (32, 18, 12)]):
        c = cases.drycbl(i, j, k, seed=110 + q, dt=2.)
        rng = np.random.default_rng(110 + q)
        for n in ("u", "v"):
            c.fields[n] = rng.normal(1., 0.3, (k, j, i))
        c.swbuffer, c.buffer_zstart, c.buffer_sigma = True, 2500., 0.01
        out.append(c)
    return out


def option(mhh, models, tmp):
    kern, _ = mhh.load()
    mhh.check(kern.mhh_ctx_set_option(models[0].ctx(), b"tendency_kernel", 0), "option")
    mhh.check(kern.mhh_ctx_set_option(models[2].ctx(), b"tdma_kernel", 1), "option")


def process_option(mhh, models, tmp):
    mhh.set_option("tendency_kernel", 0)


def layer(mhh, models, tmp):
    kern, _ = mhh.load()
    mhh.check(kern.mhh_buffer_setup(models[1].ctx(), 1000., 0.02, 1.), "buffer")


def time_step(mhh, models, tmp):
    case = made()[0]
    case.dt = 1.
    other = mhh.Model(case, precision=models[0].precision)
    other.run_steps(2)
    t = other.save(str(tmp))
    other.close()
    models[0].load(str(tmp), t)


def timing(mhh, models, tmp):
    mhh.Timing.enable(True)
    mhh.set_option("tendency_kernel", 0)


@pytest.mark.parametrize("change", [option, process_option, layer, time_step, timing], ids=lambda f: f.__name__)
@pytest.mark.parametrize("mode", [2, 3], ids=["graphs", "batched"])
def test_change_between_calls(mhh, tmp_path, mode, change):
    out = []
    for q, how in enumerate((mhh.ENS_STREAMS, mode)):
        models = [mhh.Model(c, precision=mhh.FP32) for c in made()]
        ens = mhh.Ensemble(models)
        tmp = tmp_path / str(q)
        tmp.mkdir()
        try:
            ens.run_steps(3, how)
            ens.synchronize()
            change(mhh, models, tmp)
            ens.run_steps(3, how)
            ens.synchronize()
        finally:
            mhh.set_option("tendency_kernel", -1)
            mhh.Timing.enable(False)
            mhh.Timing.reset()
        ens.run_steps(3, how)
        ens.synchronize()
        out.append([{n: m.get(n).copy() for n in ("u", "v", "w", "th")} for m in models])
        ens.close()
        for m in models:
            m.close()
    for a, b in zip(*out):
        for n in a:
            assert np.array_equal(a[n], b[n]), n
