"""The level-chunk height that the marching kernels choose per launch
(mhh::auto_kchunk), called in the built library on the CPU."""
import ctypes
import math
import random
import time

import pytest


@pytest.fixture(scope="module")
def height():
    from microhh_gb300 import build
    k, _ = build.build()
    f = getattr(ctypes.CDLL(k, mode=ctypes.RTLD_GLOBAL), "_ZN3mhh11auto_kchunkEixibi")
    f.restype = ctypes.c_int
    f.argtypes = [ctypes.c_int, ctypes.c_longlong, ctypes.c_int, ctypes.c_bool, ctypes.c_int]
    return f


def by_chunks(tiles, ktot, dbl, most, nsm=152):
    """The cheapest height over every number of chunks, the costs as stated at
    auto_kchunk."""
    best, cost = 0, 0.
    for n in range(-(-ktot // most), ktot + 1):
        kc = -(-ktot // n)
        blocks = tiles * -(-ktot // kc)
        t = math.ceil(blocks / nsm) * (kc + 3) if dbl else (tiles * ktot + 3. * blocks) / nsm + 1.25 * (kc + 3)
        if not best or t < cost:
            best, cost = kc, t
    return best


def test_height_is_the_cheapest(height):
    rng = random.Random(5)
    for _ in range(3000):
        tiles, ktot = int(math.exp(rng.uniform(0, 12))), int(math.exp(rng.uniform(0, 7)))
        dbl = rng.random() < 0.5
        assert height(0, tiles, ktot, dbl, 64) == by_chunks(tiles, ktot, dbl, 64), (tiles, ktot, dbl)


def test_requested_height(height):
    assert [height(k, 100, 300, False, 64) for k in (4, 32, 64, 128)] == [4, 32, 64, 64]


def test_tall_grids_search_no_longer(height):
    """A launch on a tall grid searches the 64 heights, not every number of
    chunks: a million levels took some milliseconds a launch, 2000 launches take
    well under a second."""
    t = time.perf_counter()
    for _ in range(2000):
        assert height(0, 1, 1000000, False, 64) == 64
    assert time.perf_counter() - t < 1.
