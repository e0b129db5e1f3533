"""A step that cannot be captured as a graph is launched kernel by kernel, and
only the kernels that ran are counted.  The failure is made on the host: a
preloaded library's cudaStreamEndCapture ends the capture, drops the graph and
returns cudaErrorStreamCaptureInvalidated, as for a call that a capture forbids."""
import json
import os
import shutil
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

FAKE = r"""
#include <dlfcn.h>
static int ended = 0;
extern "C" int ends(void) { return ended; }
extern "C" int cudaStreamEndCapture(void* stream, void** graph)
{
    void* rt = dlopen("libcudart.so.13", RTLD_LAZY | RTLD_NOLOAD);
    int (*end)(void*, void**) = (int (*)(void*, void**))dlsym(rt, "cudaStreamEndCapture");
    int (*destroy)(void*) = (int (*)(void*))dlsym(rt, "cudaGraphDestroy");
    const int rc = end(stream, graph);
    if (rc == 0 && *graph) destroy(*graph);
    *graph = nullptr;
    ++ended;
    return 901;
}
"""

RUN = r"""
import ctypes, hashlib, json, sys
import torch
import microhh_gb300 as mhh
from microhh_gb300 import cases
mhh.load()
out = {}
for fused in (True, False):
    for timed in (True, False):
        m = mhh.Model(cases.drycbl(24, 20, 16, seed=97, dt=2.), precision=64)
        n0 = mhh.launch_count()
        mhh.Timing.enable(timed)
        m.run_steps(9, fused=fused)
        m.synchronize()
        mhh.Timing.enable(False)
        mhh.Timing.reset()
        sums = [hashlib.md5(m.get(n).tobytes()).hexdigest() for n in ("u", "v", "w", "th")]
        out[f"{fused} {timed}"] = [mhh.launch_count() - n0, sums]
        m.close()
out["ends"] = ctypes.CDLL(sys.argv[1]).ends()
print(json.dumps(out))
"""


def test_failed_capture(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("no C++ compiler")
    src, lib = tmp_path / "fake.cpp", tmp_path / "libfake.so"
    src.write_text(FAKE)
    subprocess.run(["g++", "-shared", "-fPIC", str(src), "-o", str(lib), "-ldl"], check=True)
    env = dict(os.environ, LD_PRELOAD=str(lib), PYTHONPATH=ROOT)
    r = subprocess.run([sys.executable, "-c", RUN, str(lib)], env=env, cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    out = json.loads(r.stdout.strip().splitlines()[-1])
    assert out["ends"] == 2, out["ends"]        # one capture tried per model, and not again
    for fused in (True, False):
        assert out[f"{fused} False"] == out[f"{fused} True"], fused
