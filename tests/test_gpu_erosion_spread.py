"""The one-lane erosion kernel with fewer than 32 droplets per warp, from one to all, over the counts where
their number changes: droplets that never meet follow the serial oracle in the kernel's own precision
(among thousands, one or two take a step the other way in FP64), all droplets are eroded (mass
balance), and a warp's last, partly filled group is too."""
import numpy as np
import pytest

import helpers
from test_gpu_erosion import erode_runs, terrain

pytestmark = pytest.mark.gpu

WARPS = 24 * 152  # of a launch before its warps take more droplets


@pytest.mark.parametrize("count", [1, 31, 400, WARPS, WARPS + 1, 2 * WARPS + 1])
def test_droplets_that_never_meet_follow_the_oracle(dev, oracle, stpgb, count):
    side = 44 * int(np.ceil(np.sqrt(count))) + 40  # starts 44 px apart, 16 steps, brush reach 3
    h = terrain(side, side, 4)
    g = np.arange(int(np.ceil(np.sqrt(count))), dtype=np.float32) * 44 + 30.37
    starts = np.stack(np.meshgrid(g, g), 2).reshape(-1, 2)[:count].astype(np.float32).ravel()
    s = helpers.raindrop_dict(count, radius=3, lifetime=16)
    idx, w = oracle.brush(side, 3)
    ref, ref_res, _ = oracle.erode(h, s, starts, idx, w, fp64=False)
    [(out, res)] = erode_runs(dev, stpgb, h, (side, side), (1, 1), s, starts, 1, lanes=1, pointwise=True)
    rms = float(np.sqrt(np.mean((out - ref.astype(np.float64)) ** 2)))
    assert rms <= 1e-5 * float(h.max() - h.min()), rms
    assert abs(res - ref_res) <= 1e-4 * max(ref_res, 1e-6) + 1e-6
    assert not np.array_equal(out, h)


@pytest.mark.parametrize("count", [4 * WARPS + 3, 8 * WARPS + 1, 16 * WARPS, 16 * WARPS + 1, 32 * WARPS + 77])
def test_every_droplet_is_eroded(dev, oracle, stpgb, count):
    side = 512
    h = terrain(side, side, 5)
    starts = np.random.default_rng(count).uniform(4, side - 5, 2 * count).astype(np.float32)
    s = helpers.raindrop_dict(count, radius=2, lifetime=10)
    before = h.astype(np.float64).sum()
    [(out, res)] = erode_runs(dev, stpgb, h, (side, side), (1, 1), s, starts, 1, lanes=1, pointwise=True)
    assert np.isfinite(out).all() and not np.array_equal(out, h)
    assert abs((before - out.sum()) - res) <= 1e-5 * before
    # the last droplets alone change the map too: they are in the last, partly filled warp
    last = starts[-2:]
    [(one, _)] = erode_runs(dev, stpgb, h, (side, side), (1, 1), dict(s), last, 1, lanes=1, pointwise=True)
    x, y = int(last[0]), int(last[1])
    window = np.s_[max(y - 2, 0):y + 3, max(x - 2, 0):x + 3]
    assert np.array_equal(one[window], h[window]) or not np.array_equal(out[window], h[window])
