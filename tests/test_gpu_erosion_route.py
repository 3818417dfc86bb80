"""Which kernels erode a call.  Droplets that never meet leave the same bits run after run, and the tiles,
which hold heights as integers, other bits than the kernels on the L2: a call that the tiles erode
differs from those, and one that they do not take equals them bit for bit.  (How near either is to the
oracle: tests/test_gpu_erosion_tiles.py, tests/test_gpu_erosion.py.)"""
import ctypes as C

import numpy as np
import pytest

import helpers
from test_gpu_erosion import terrain
from test_gpu_erosion_accuracy import POINTWISE, TILES, erode, on_the_l2
from test_gpu_erosion_tiles import erode as erode_tiles
from test_gpu_erosion_tiles import sparse_starts

pytestmark = pytest.mark.gpu

EXACT = 1


@pytest.mark.parametrize("size,brush,first", [
    ((332, 284), 1, 0), ((332, 284), 2, 0), ((332, 284), 3, 0), ((332, 284), 4, 17), ((1500, 41), 5, 17),
    ((44, 900), 6, 17), ((40, 40), 4, 17), ((80, 81), 3, 17), ((332, 284), 6, 23)])
def test_the_flag_takes_the_tiles(dev, stpgb, size, brush, first):
    h = terrain(*size, brush)
    s = helpers.raindrop_dict(1, radius=brush, lifetime=14)
    starts = sparse_starts(*size, 41.0, first)
    out = erode(stpgb, h, size, (1, 1), s, starts, flags=TILES)
    assert np.array_equal(out, erode(stpgb, h, size, (1, 1), s, starts, flags=TILES))
    ref = on_the_l2(stpgb, h, size, (1, 1), s, starts)
    assert not np.array_equal(ref, h)
    assert np.array_equal(ref, on_the_l2(stpgb, h, size, (1, 1), s, starts))
    assert not np.array_equal(out, ref)


@pytest.mark.parametrize("case", ["peak", "outlier", "nan", "infinite", "zero", "wide brush", "long life", "radius", "captured"])
def test_what_the_tiles_leave_to_the_l2(dev, oracle, stpgb, case):
    """One cell above 8 times the mean height, 10^6 times, a NaN, an infinity, a map of zeros, a brush that
    reaches further than its radius, more than 1024 steps, a radius above 6 and a captured stream."""
    n = 328
    h = terrain(n, n, 7)
    s = helpers.raindrop_dict(1, radius=7 if case == "radius" else 3, lifetime=1100 if case == "long life" else 14)
    starts = sparse_starts(n, n, 41.0).reshape(-1, 2)
    starts = starts[np.abs(starts - 164.0).max(1) > 30.0]
    h[164, 164] = {"peak": 6.0, "outlier": 1e6, "nan": np.nan, "infinite": np.inf}.get(case, h[164, 164])
    if case == "zero":
        h[:] = 0.0
    brush = stpgb.erosion_brush(n, s["ErosionBrushRadius"])
    if case == "wide brush":
        brush = brush[0].copy(), brush[1]
        brush[0][np.argmax(brush[0])] = 5 * n
    starts = starts[(starts > 30.0).all(1) & (starts < n - 30.0).all(1)].ravel()
    if case == "long life":
        starts = starts[:2]  # it goes far, and alone
    tiles, _ = erode_tiles(stpgb, h, (n, n), (1, 1), s, starts, brush=brush, stream=case, check=False)

    # the same call without the flag, which is small
    L, ptr = stpgb.lib(), lambda t: C.c_void_p(t.data_ptr())
    import torch
    d, st = torch.from_numpy(h).cuda(), torch.from_numpy(starts).cuda()
    idx, w = (torch.from_numpy(a).cuda() for a in brush)
    info, rain = stpgb.NNInfo.make((n, n), (1, 1)), stpgb.RaindropSetting(**s)
    stpgb.check(L.stpgb_hydraulic_erosion_ex(ptr(d), C.byref(info), C.byref(rain), ptr(st), len(starts) // 2, ptr(idx),
                                             ptr(w), len(idx), None, None, 0, 1, 0,
                                             C.c_void_p(torch.cuda.current_stream().cuda_stream)))
    out = d.cpu().numpy()
    assert np.array_equal(tiles, out, equal_nan=True)
    assert case == "zero" or not np.array_equal(out, h, equal_nan=True)


@pytest.mark.parametrize("lanes,flags", [(0, POINTWISE), (0, EXACT), (1, 0), (2, 0), (4, POINTWISE)])
def test_lanes_and_other_flags_override_the_tiles(dev, stpgb, lanes, flags):
    n = 328
    h = terrain(n, n, 5)
    s = helpers.raindrop_dict(1, radius=3, lifetime=14)
    starts = sparse_starts(n, n, 41.0)
    out = erode(stpgb, h, (n, n), (1, 1), s, starts, lanes=lanes, flags=flags | TILES)
    assert np.array_equal(out, erode(stpgb, h, (n, n), (1, 1), s, starts, lanes=lanes, flags=flags))
    assert not np.array_equal(out, erode(stpgb, h, (n, n), (1, 1), s, starts, flags=TILES))


def test_default_of_large_calls(dev, stpgb):
    """9216 droplets of 1000 steps and 109 points, 48 px apart on hills whose foot is flat, where a droplet
    without inertia ends: 10^9 points that could be eroded, and no two droplets that meet.  Of 900 steps
    the points are fewer, and as the neighbourhood of a chunk of 932^2 the start area is below 2^20."""
    k, apart, n = 96, 48, 4660
    g = np.arange(k) * apart + 30
    y, x = np.mgrid[0:n, 0:n].astype(np.float32)
    from_hill = [(a - 30 + apart // 2) % apart - apart // 2 for a in (x, y)]
    h = (0.5 + 0.03 * np.clip(1 - np.hypot(*from_hill) / 9, 0, None)).astype(np.float32)
    starts = np.stack(np.meshgrid(g + 2.37, g + 1.61), 2).reshape(-1, 2)
    starts = (starts + np.random.default_rng(1).uniform(-0.3, 0.3, starts.shape)).astype(np.float32).ravel()
    for lifetime, S, nn, tiles in ((1000, n, 1, True), (900, n, 1, False), (1000, n // 5, 5, False)):
        s = helpers.raindrop_dict(1, radius=6, lifetime=lifetime)
        s["Inertia"] = 0.0
        assert (len(starts) // 2 * lifetime * len(stpgb.erosion_brush(n, 6)[0]) >= 10**9) == (lifetime == 1000)
        out = erode(stpgb, h, (S, S), (nn, nn), s, starts)
        assert np.array_equal(out, erode(stpgb, h, (S, S), (nn, nn), s, starts, flags=TILES)) == tiles
        assert np.array_equal(out, on_the_l2(stpgb, h, (S, S), (nn, nn), s, starts)) == (not tiles)
