"""The drop-in generator's chunk arrays by the copies that go one after the other: arrays at odd
addresses, as those at even ones, and an array that stands for two places of the neighbourhood, which
the later place's heights are left in."""
import numpy as np
import pytest

import helpers

pytestmark = pytest.mark.gpu


def odd(a):
    """A copy of `a` at an odd address."""
    raw = np.zeros(a.nbytes + 2, np.uint8)
    start = 1 - raw.ctypes.data % 2
    view = raw[start:start + a.nbytes].view(a.dtype).reshape(a.shape)
    view[:] = a
    assert view.ctypes.data % 2 == 1
    return view


def generator(stpgb, size, radius, brush=2):
    rain = stpgb.RaindropSetting(**helpers.raindrop_dict(10, radius=brush, lifetime=20))
    return stpgb.STPHeightfieldGenerator(stpgb.ChunkSetting(size, (3, 3), (3, 3)), rain,
                                         stpgb.SimplexSetting(9, 8, 0.25), helpers.biome_table(5, 3), radius)


def chunks_of(whole, w, h):
    return [np.ascontiguousarray(whole[y * h:(y + 1) * h, x * w:(x + 1) * w]) for y in range(3) for x in range(3)]


@pytest.mark.parametrize("size,radius", [((64, 48), 16), ((37, 23), 8)])
def test_odd_addresses(stpgb, dev, oracle, size, radius):
    w, h = size
    gen = generator(stpgb, size, radius)
    chunks = chunks_of(oracle.voronoi(3 * w, 3 * h, (-w, -h), 11, 5, 9), w, h)
    out, ref = np.zeros((h, w), np.float32), np.zeros((h, w), np.float32)
    gen.generate(ref, chunks, (100.0, -40.0))
    gen.generate(out, [odd(c) for c in chunks], (100.0, -40.0))
    assert np.array_equal(out, ref)
    heights = [np.random.default_rng(n).random((h, w), np.float32) for n in range(9)]
    shifted, fixed = [odd(c) for c in heights], [odd(np.zeros((h, w), np.uint16)) for _ in range(9)]
    assert gen.erode(shifted, fixed, np.zeros(0, np.float32)) == 0.0
    for a, b, f in zip(shifted, heights, fixed):
        assert np.array_equal(a, b) and np.array_equal(f, oracle.format(b))


@pytest.mark.parametrize("first", [0, 5])
def test_an_array_for_two_places(stpgb, dev, first):
    """A droplet that leaves the middle chunk for the last one: place `first` has the last one's array."""
    w = h = 64
    gen = generator(stpgb, (w, h), 16)
    y, x = np.mgrid[0:h, 0:w]
    slope = (0.9 - 0.002 * (x + y)).astype(np.float32)
    heights = [slope - np.float32(0.002 * (n % 3 * w + n // 3 * h)) for n in range(9)]
    starts = np.array([2 * w - 4.3, 2 * h - 4.6], np.float32)

    def run(shared):
        arrays = [c.copy() for c in heights]
        fixed = [np.zeros((h, w), np.uint16) for _ in range(9)]
        arrays[first][:] = arrays[8]
        if shared:
            arrays[first], fixed[first] = arrays[8], fixed[8]
        gen.erode(arrays, fixed, starts)
        return arrays, fixed

    (a, fa), (b, fb) = run(False), run(True)
    assert not np.array_equal(a[8], a[first])
    for n in range(9):
        if n != first:
            assert np.array_equal(a[n], b[n]) and np.array_equal(fa[n], fb[n]), n
