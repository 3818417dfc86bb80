"""Noise far outside the range of its samples' cells: octaves whose frequency overflows and biomes of scale
0, whose samples lie at infinity, where every corner is out of reach.  The heights are the FP32
oracle's, the noise's tolerance allowed."""
import numpy as np
import pytest

import helpers

pytestmark = pytest.mark.gpu

NOISE_TOL = 2e-6


@pytest.mark.parametrize("scale,octave,lacunarity", [
    (50.0, 100, 2.0), (50.0, 126, 2.0), (50.0, 135, 2.0), (50.0, 200, 2.0), (50.0, 40, 10.0), (0.0, 3, 2.0), (1e-37, 4, 2.0)])
def test_heights_at_overflowing_samples(dev, oracle, stpgb, scale, octave, lacunarity):
    import torch
    mx, my = 48, 36
    perm, grad = stpgb.permutation_generate(42, 8, 0.2181661565)
    table = np.zeros(1, stpgb.BIOME_DTYPE)
    table[0] = (scale, octave, 0.5, lacunarity, 0.25, 1.0)
    off = np.arange(mx * my + 1, dtype=np.uint32)
    bins = np.zeros(mx * my, stpgb.BIN_DTYPE)
    bins["Weight"] = 1.0
    where = (1000.25, -2000.75)  # no sample at 0, whose product with an infinite frequency is no number
    ref = oracle.multibiome(off, bins, table, perm, grad, (mx, my), where)
    assert ref.min() >= 0.25
    out = torch.zeros((my, mx), device="cuda")
    dev.multibiome_heightmap(out, mx, torch.from_numpy(off.view(np.int32)).cuda(),
                             torch.from_numpy(bins.view(np.int64)).cuda(), (mx, my), where,
                             torch.from_numpy(perm).cuda(), torch.from_numpy(grad).cuda(),
                             torch.from_numpy(table.view(np.float32)).cuda())
    assert np.abs(out.cpu().numpy() - ref).max() <= NOISE_TOL
