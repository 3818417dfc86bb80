"""Erosion in shared-memory tiles (STPGB_EROSION_TILES, and the default of large calls).

Droplets that never meet follow the FP64 serial oracle within the bound of the other kernels
(tests/test_gpu_erosion.py: per-pixel RMS below 1e-5 of the height range), whichever tile edges they
cross: the tiles' unit is below 2^-25 of the largest height, and what differs beyond that is a path
through a cell edge.  Racing droplets conserve mass within 1e-5.  Maps, brushes and streams that the
tiles do not take keep to the other kernels."""
import ctypes as C

import numpy as np
import pytest

import helpers
from test_gpu_erosion import terrain

pytestmark = pytest.mark.gpu

TILES = 4


def erode(stpgb, h, map_size, nn, setting, starts, brush=None, stream=None, check=True):
    """stpgb_hydraulic_erosion_ex with STPGB_EROSION_TILES; (map, residual)."""
    import torch
    d = torch.from_numpy(np.ascontiguousarray(h, np.float32)).cuda()
    st = torch.from_numpy(np.ascontiguousarray(starts, np.float32)).cuda()
    idx, w = brush if brush else stpgb.erosion_brush(h.shape[1], setting["ErosionBrushRadius"])
    d_idx, d_w = torch.from_numpy(idx).cuda(), torch.from_numpy(w).cuda()
    res = torch.zeros(1, dtype=torch.float64, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    info, rd = stpgb.NNInfo.make(map_size, nn), stpgb.RaindropSetting(**setting)
    ptr = lambda t: C.c_void_p(t.data_ptr())

    def call(s):
        stpgb.check(stpgb.lib().stpgb_hydraulic_erosion_ex(ptr(d), C.byref(info), C.byref(rd), ptr(st), len(starts) // 2,
                                                           ptr(d_idx), ptr(d_w), len(idx), ptr(res), ptr(status), 0, 1,
                                                           TILES, C.c_void_p(s)))
    if stream == "captured":
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            call(torch.cuda.current_stream().cuda_stream)
        graph.replay()
    else:
        call(torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    if check:
        assert int(status.item()) == 0
    return d.cpu().numpy(), float(res.item())


def sparse_starts(mx, my, spacing, first=0):
    xs, ys = np.meshgrid(np.arange(first + 0.37, mx - 1, spacing), np.arange(first + 0.61, my - 1, spacing))
    return np.stack([xs.ravel(), ys.ravel()], 1).ravel().astype(np.float32)


@pytest.mark.parametrize("size,brush,first", [
    ((331, 283), 1, 0), ((331, 283), 2, 0), ((332, 284), 3, 0), ((331, 283), 4, 0), ((1500, 41), 5, 0),
    ((41, 900), 6, 0), ((40, 40), 4, 0), ((80, 81), 3, 0), ((1500, 41), 5, 17), ((41, 900), 6, 17), ((40, 40), 4, 17),
    ((80, 81), 3, 17), ((331, 283), 5, 23), ((332, 284), 6, 23)])
def test_sparse_droplets_follow_the_oracle_across_tiles(dev, oracle, stpgb, size, brush, first):
    """Starts 41 px apart, one off the tiles' side, and 14 steps of one pixel, so no two brushes meet
    (14 + 14 + 2 * 6 < 41); maps odd and even, as small as one tile and as narrow as one."""
    mx, my = size
    h = terrain(mx, my, brush)
    s = helpers.raindrop_dict(1, radius=brush, lifetime=14)
    starts = sparse_starts(mx, my, 41.0, first)
    out, res = erode(stpgb, h, size, (1, 1), s, starts)
    idx, w = oracle.brush(mx, brush)
    ref, ref_res, _ = oracle.erode(h, s, starts, idx, w, fp64=True)
    rms = float(np.sqrt(np.mean((out.astype(np.float64) - ref) ** 2)))
    assert rms <= 1e-5 * float(h.max() - h.min()), rms
    assert abs(res - ref_res) <= 1e-4 * max(ref_res, 1e-6) + 1e-6


@pytest.mark.parametrize("S,nn,density,brush,lifetime", [
    (64, 3, 2.3, 3, 30), (96, 3, 1.0, 5, 64), (101, 1, 0.9, 4, 50), (48, 5, 7.0, 2, 40), (200, 3, 2.0, 6, 50)])
def test_racing_droplets_conserve_mass(dev, oracle, stpgb, S, nn, density, brush, lifetime):
    h = terrain(nn * S, nn * S, S)
    count = int(density * S * S)
    s = helpers.raindrop_dict(count, radius=brush, lifetime=lifetime)
    starts = oracle.droplet_starts(count, 9, 0, (S, S), (nn, nn))
    out, res = erode(stpgb, h, (S, S), (nn, nn), s, starts)
    total = h.astype(np.float64).sum()
    assert abs((total - out.astype(np.float64).sum()) - res) <= 1e-5 * total
    assert np.isfinite(out).all() and out.min() >= h.min() - 1e-3 and out.max() <= h.max() + 1e-3


def test_droplets_that_start_together_conserve_mass(dev, stpgb):
    """Every droplet from one place: each takes and puts on the same cells as the others."""
    h = terrain(192, 192, 3)
    count = 6000
    s = helpers.raindrop_dict(count, radius=4, lifetime=50)
    starts = np.tile(np.array([90.3, 101.8], np.float32), count)
    out, res = erode(stpgb, h, (64, 64), (3, 3), s, starts)
    total = h.astype(np.float64).sum()
    assert np.isfinite(out).all()
    assert abs((total - out.astype(np.float64).sum()) - res) <= 1e-5 * total


@pytest.mark.parametrize("case", ["outlier", "nan", "infinite", "zero", "wide brush", "captured"])
def test_what_the_tiles_do_not_take(dev, oracle, stpgb, case):
    """One cell 10^6 times the others', a NaN, an infinity, a map of zeros, a brush that reaches further
    than its radius, and a captured stream: sparse droplets away from the odd cell erode as the oracle's,
    through the kernels that keep the map in global memory."""
    n, spacing = 328, 41.0
    h = terrain(n, n, 7)
    if case == "zero":
        h[:] = 0.0
    s = helpers.raindrop_dict(1, radius=3, lifetime=14)
    starts = sparse_starts(n, n, spacing).reshape(-1, 2)
    odd = {"outlier": 1e6, "nan": np.nan, "infinite": np.inf}.get(case)
    if odd is not None:
        starts = starts[np.abs(starts - 164.0).max(1) > 30.0]
        h[164, 164] = odd
    starts = starts.ravel()
    brush = oracle.brush(n, 3)
    if case == "wide brush":
        at = oracle.brush(n, 6)
        keep = [i for i, v in enumerate(at[0]) if v in (0, 5, -5, 5 * n)]
        brush = at[0][keep].copy(), np.full(len(keep), 0.25, np.float32)
        starts = starts.reshape(-1, 2)
        starts = starts[(starts > 30.0).all(1) & (starts < n - 30.0).all(1)].ravel()
    out, res = erode(stpgb, h, (n, n), (1, 1), s, starts, brush=brush, stream=case)
    same = np.isfinite(h)
    ref, ref_res, _ = oracle.erode(np.where(same, h, 0.5).astype(np.float32), s, starts, *brush, fp64=True)
    assert np.array_equal(out[~same], h[~same], equal_nan=True)
    if case == "outlier":
        same[164, 164] = False
        assert out[164, 164] == h[164, 164]
    rms = float(np.sqrt(np.mean((out[same].astype(np.float64) - ref[same]) ** 2)))
    assert rms <= 1e-5 * max(float(h[same].max() - h[same].min()), 1e-3), rms
    assert abs(res - ref_res) <= 1e-4 * max(ref_res, 1e-6) + 1e-6


def test_default_of_a_large_call_takes_the_tiles(dev, oracle, stpgb):
    """At 10^9 brush points and more (here 420,000 droplets of 50 steps and 69 points, an odd width, a
    stream of its own) the default call is the tiles'."""
    import torch
    S, count = 401, 420000
    h = terrain(3 * S, 3 * S, 5)
    s = helpers.raindrop_dict(count, radius=5, lifetime=50)
    starts = oracle.droplet_starts(count, 3, 0, (S, S), (3, 3))
    d = torch.from_numpy(h).cuda()
    idx, w = stpgb.erosion_brush(3 * S, 5)
    res = torch.zeros(1, dtype=torch.float64, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        dev.hydraulic_erosion(d, (S, S), (3, 3), stpgb.RaindropSetting(**s), torch.from_numpy(starts).cuda(), count,
                              torch.from_numpy(idx).cuda(), torch.from_numpy(w).cuda(), res, status)
        dev.status_check(status)
    out = d.cpu().numpy()
    total = h.astype(np.float64).sum()
    assert abs((total - out.astype(np.float64).sum()) - float(res.item())) <= 1e-5 * total
    assert np.isfinite(out).all() and out.min() >= h.min() - 1e-3 and out.max() <= h.max() + 1e-3
