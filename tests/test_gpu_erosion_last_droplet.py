"""The one-lane erosion kernel's last, partly filled warp: the launch's last droplet starts where none of the
others comes, and its cells are as its own oracle's.  The counts lie where a warp's droplets change, by
the device's own number of SMs."""
import numpy as np
import pytest

import helpers
from test_gpu_erosion import erode_runs, terrain

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("per_sm,more", [(0, 1), (24, 1), (48, 1), (96, 3), (192, 1), (384, 0), (384, 1), (768, 77)])
def test_the_last_droplet_is_eroded(dev, oracle, stpgb, per_sm, more):
    import torch
    count = per_sm * torch.cuda.get_device_properties(0).multi_processor_count + more
    side = 512
    h = terrain(side, side, 5)
    s = helpers.raindrop_dict(count, radius=2, lifetime=10)
    others = np.random.default_rng(count).uniform(4, side - 5, (count - 1, 2))
    others[:, 0] *= 0.8  # 10 steps and a brush of 2 keep them left of 425
    last = np.array([[480.4, 250.7]])
    starts = np.concatenate([others, last]).astype(np.float32).ravel()
    [(out, _)] = erode_runs(dev, stpgb, h, (side, side), (1, 1), s, starts, 1, lanes=1, pointwise=True)
    ref, _, _ = oracle.erode(h, s, last.astype(np.float32).ravel(), *oracle.brush(side, 2), fp64=False)
    right = np.s_[:, 440:]
    assert not np.array_equal(ref[right], h[right])
    assert np.abs(out[right] - ref[right]).max() <= 1e-5 * float(h.max() - h.min())
    assert np.array_equal(out[right] != h[right], ref[right] != h[right])
