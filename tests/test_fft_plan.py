"""The plans of the run-time-plan transforms (mhh_fft_plan.h, compiled here) on
the CPU: every length that a block's shared memory holds, and the index algebra
of the stages (mhh_pres.cu: fg_stage, fe_stage) restated in numpy."""
import os
import shutil
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "microhh_gb300", "csrc")
# 200 KB for two buffers and the twiddles of one pair of sequences.
LONGEST = {64: 200 * 1024 // 48, 32: 200 * 1024 // 24}
PAIRS = {0x32, 0x52, 0x24, 0x33, 0x34}

MAIN = r"""
#include <cstdio>
#include "mhh_fft_plan.h"
int main()
{
    for (int n=2; n<=8533; ++n)
    {
        int r = n;
        for (int f : {2, 3, 5, 7}) while (r % f == 0) r /= f;
        if (r != 1) continue;
        int fac[64];
        for (int prec : {64, 32})
        {
            const int m = prec == 64 ? mhh::plan_radices(n, fac) : mhh::plan_floats(n, fac);
            std::printf("%d %d", n, prec);
            for (int q=0; q<m; ++q) std::printf(" %d", fac[q]);
            std::printf("\n");
        }
    }
}
"""


@pytest.fixture(scope="module")
def plans(tmp_path_factory):
    cxx = os.environ.get("CXX", "g++")
    if shutil.which(cxx) is None:
        pytest.skip("no C++ compiler")
    d = tmp_path_factory.mktemp("plan")
    (d / "main.cpp").write_text(MAIN)
    subprocess.run([cxx, "-std=c++17", "-O1", "-I" + CSRC, str(d / "main.cpp"), "-o", str(d / "plan")], check=True)
    out = {}
    for line in subprocess.run([str(d / "plan")], check=True, capture_output=True, text=True).stdout.splitlines():
        n, prec, *codes = map(int, line.split())
        out[n, prec] = codes
    return out


def parts(code, prec):
    """(RA, B, in frequency) of a stage."""
    if prec == 64:
        return code, 1, False
    return code & 15, max(code >> 4, 1), code >> 4 == 0


def test_every_length(plans):
    for (n, prec), codes in plans.items():
        if n > LONGEST[prec]:
            continue
        assert len(codes) <= 8, (n, prec, codes)       # eight codes of eight bits
        p = 1
        for q, code in enumerate(codes):
            if prec == 64:
                assert 2 <= code <= 10, (n, codes)
            else:
                assert code in PAIRS or code in (0x12, 0x13, 0x14, 0x15, 0x17, 0x18, 8) or (q == 0 and code in (2, 4)), (n, codes)
            ra, b, dif = parts(code, prec)
            R = ra * b
            assert (n // p) % R == 0, (n, prec, codes)
            T = n // R
            step = T // p
            # The largest twiddle indexes of the stage.
            if dif:
                # No twiddles in the last stage, where p = T.
                assert p == T or (ra - 1) * (T - 1 - (T - 1) % p) < n
            else:
                assert (ra - 1) * (p - 1) * b * step < n
                assert (b - 1) * (p - 1 + (ra - 1) * p) * step < n
            p *= R
        assert p == n, (n, prec, codes)


def dft(u):
    R = u.shape[0]
    k = np.arange(R)
    return np.tensordot(np.exp(-2j * np.pi * np.outer(k, k) / R), u, 1)


def transform(x, codes, prec):
    n = len(x)
    w = np.exp(-2j * np.pi * np.arange(n) / n)
    src, p = x.astype(complex), 1
    for code in codes:
        ra, b, dif = parts(code, prec)
        T = n // (ra * b)
        step = T // p
        i = np.arange(T)
        k = i % p
        dst = np.full(n, np.nan, complex)
        j = (i - k) * ra * b + k
        u = np.empty((b, ra, T), complex)
        for r in range(b):
            for a in range(ra):
                u[r, a] = src[i + (r + a * b) * T]
                if not dif and a:
                    u[r, a] *= w[a * k * b * step]
            u[r] = dft(u[r])
        if dif:
            for a in range(ra):
                dst[j + a * p] = u[0, a] * (w[a * (i - k)] if a and p != T else 1.)
        else:
            for m in range(ra):
                v = u[:, m].copy()
                for r in range(1, b):
                    v[r] *= w[r * (k + m * p) * step]
                v = dft(v)
                for r in range(b):
                    dst[j + (m + ra * r) * p] = v[r]
        src, p = dst, p * ra * b
    return src


@pytest.mark.parametrize("prec", [64, 32])
def test_stages_are_the_transform(plans, prec):
    """Within 8 eps n of the largest value (a bound of any ordering's sum)."""
    rng = np.random.default_rng(3)
    for (n, q), codes in plans.items():
        if q != prec or (n > 600 and n not in (720, 768, 1000, 1024, 1536, 2048, 2187, 2401, 3125, 4096)):
            continue
        x = rng.standard_normal(n) + 1j * rng.standard_normal(n)
        want = np.fft.fft(x)
        got = transform(x, codes, prec)
        assert np.abs(got - want).max() <= 8 * 2.3e-16 * n * np.abs(want).max(), (n, codes)


def test_float_radices_of_a_length(plans):
    """The elementary radices of float lengths, which with their order fix the
    rounding of every float field: lengths of each rule."""
    want = {32: [8, 4], 48: [8, 2, 3], 128: [2, 8, 8], 512: [8, 8, 8], 1024: [8, 8, 8, 2], 120: [4, 2, 3, 5],
            1536: [4, 4, 4, 4, 2, 3], 2048: [4, 4, 4, 4, 4, 2], 150: [2, 3, 5, 5], 189: [3, 3, 3, 7]}
    got = {n: [r for c in plans[n, 32] for r in ((c & 15, c >> 4) if c >> 4 > 1 else (c & 15,))] for n in want}
    assert got == want
