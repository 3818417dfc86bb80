"""Launches whose blocks take several strips of pixels (heights) or several tiles (splatmap), so that
they share the noise's tables: sizes that leave partial strips, rows that wrap within a strip and
partial tiles, against the oracle with the tolerances of test_gpu_noise.py and test_gpu_splat.py."""
import numpy as np
import pytest

import helpers
from test_gpu_noise import NOISE_TOL
from test_gpu_splat import SIMPLEX, near_boundary
from test_splat import DEMO_ALTITUDE, DEMO_GRADIENT

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("map_size", [(641, 633), (3, 150001), (400003, 1), (1, 390001), (1531, 1537)])
def test_heights_of_several_strips(dev, oracle, stpgb, map_size):
    import torch
    mx, my = map_size
    n = mx * my
    rng = np.random.default_rng(mx)
    counts = rng.integers(1, 3, n)
    off = np.zeros(n + 1, np.uint32)
    off[1:] = np.cumsum(counts)
    bins = np.zeros(int(off[-1]), stpgb.BIN_DTYPE)
    bins["Item"] = rng.integers(0, 4, len(bins))
    bins["Weight"] = np.repeat(1.0 / counts, counts).astype(np.float32)
    perm, grad = stpgb.permutation_generate(11, 8, 0.2181661565)
    table = helpers.biome_table(4, 11)
    ref = oracle.multibiome(off, bins, table, perm, grad, map_size, (77.0, -1300.0))
    out = torch.full((my, mx), float("nan"), device="cuda")
    dev.multibiome_heightmap(out, mx, torch.from_numpy(off.view(np.int32)).cuda(),
                             torch.from_numpy(np.ascontiguousarray(bins).view(np.int64)).cuda(), map_size,
                             (77.0, -1300.0), torch.from_numpy(perm).cuda(), torch.from_numpy(grad).cuda(),
                             torch.from_numpy(table.view(np.float32)).cuda())
    got = out.cpu().numpy()
    assert np.isfinite(got).all()
    assert np.abs(got.astype(np.float64) - ref.astype(np.float64)).max() <= NOISE_TOL


@pytest.mark.parametrize("map_size,nx,ny", [((1136, 1117), 1, 1), ((416, 405), 3, 3), ((2000, 1990), 1, 1)])
def test_splatmap_of_several_tiles(dev, oracle, stpgb, map_size, nx, ny):
    import torch
    sx, sy = map_size
    W, H = nx * sx, ny * sy
    rng = np.random.default_rng(sx)
    y, x = np.mgrid[0:H, 0:W]
    h = 0.45 + 0.3 * np.sin(x / 11.0) * np.cos(y / 13.0) + 0.12 * np.sin((x + 2 * y) / 5.0) + 0.02 * rng.random((H, W))
    hm = np.round(np.clip(h, 0, 1) * 65535).astype(np.uint16)
    bm = rng.integers(0, 3, (H // 40 + 1, W // 40 + 1)).astype(np.uint16)[y // 40, x // 40]
    chunks = [(c % nx, c // nx, float(c % nx * sx + 500), float(c // nx * sy - 90)) for c in range(nx * ny)]
    gen = stpgb.STPSplatmapGenerator(DEMO_ALTITUDE, DEMO_GRADIENT, stpgb.SimplexSetting(*SIMPLEX), map_size)
    out = torch.full((H, W), 0x77, dtype=torch.uint8, device="cuda")
    slope = torch.full((H, W), float("nan"), device="cuda")
    alt = torch.full((H, W), float("nan"), device="cuda")
    gen(torch.from_numpy(bm.view(np.int16)).cuda(), torch.from_numpy(hm.view(np.int16)).cuda(), W, out, W, W, H, chunks,
        slope, alt)
    perm, grad = stpgb.permutation_generate(*SIMPLEX)
    want, ws, wa = oracle.splatmap(bm, hm, chunks, map_size, DEMO_ALTITUDE, DEMO_GRADIENT, perm, grad)
    assert np.abs(slope.cpu().numpy() - ws).max() <= 1e-5
    assert np.abs(alt.cpu().numpy() - wa).max() <= 1e-6
    diff = out.cpu().numpy() != want
    assert not np.any(diff & ~near_boundary(ws, wa, DEMO_ALTITUDE, DEMO_GRADIENT, eps=1e-5))
    assert diff.mean() < 1e-4
