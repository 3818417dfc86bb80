"""The drop-in generator's chunk arrays, moved between host and device by one kernel: odd sizes, arrays
at odd 2-byte addresses, radii up to the whole neighbour; the heights equal the device calls' exactly
(the same kernels on the same samples), and erosion by no droplets returns every chunk as it was."""
import numpy as np
import pytest

import helpers

pytestmark = pytest.mark.gpu


def unaligned(a):
    """A contiguous copy of `a` that starts one 2-byte (float: 4-byte) element past an aligned address."""
    raw = np.zeros(a.size + 9, a.dtype)
    start = 1 + (-raw.ctypes.data // a.itemsize) % 8
    view = raw[start:start + a.size].reshape(a.shape)
    view[:] = a
    return view


@pytest.mark.parametrize("size,radius,shift", [((64, 48), 16, False), ((37, 23), 8, True), ((33, 40), 32, True),
                                               ((8, 8), 8, False), ((130, 7), 6, True)])
def test_generate_equals_device_calls(stpgb, dev, oracle, size, radius, shift):
    import torch
    w, h = size
    table = helpers.biome_table(5, 3)
    whole = oracle.voronoi(3 * w, 3 * h, (-w, -h), 11, 5, 9)
    chunks = [np.ascontiguousarray(whole[y * h:(y + 1) * h, x * w:(x + 1) * w]) for y in range(3) for x in range(3)]
    if shift:
        chunks = [unaligned(c) for c in chunks]
    rain = stpgb.RaindropSetting(**helpers.raindrop_dict(10, radius=1, lifetime=5))
    gen = stpgb.STPHeightfieldGenerator(stpgb.ChunkSetting(size, (3, 3), (3, 3)), rain,
                                        stpgb.SimplexSetting(9, 8, 0.25), table, radius)
    out = np.zeros((h, w), np.float32)
    gen.generate(out, chunks, (100.0, -40.0))
    off, bins, status = dev.shf_filter(torch.from_numpy(whole.view(np.int16)).cuda(), size, (3, 3), radius, max_items=5)
    dev.status_check(status)
    perm, grad = stpgb.permutation_generate(9, 8, 0.25)
    ref = torch.empty((h, w), device="cuda")
    dev.multibiome_heightmap(ref, w, off, bins, size, (100.0, -40.0), torch.from_numpy(perm).cuda(),
                             torch.from_numpy(grad).cuda(), torch.from_numpy(table.view(np.float32)).cuda())
    assert np.array_equal(out, ref.cpu().numpy())

    rng = np.random.default_rng(1)
    heights = [unaligned(rng.random((h, w), np.float32)) for _ in range(9)]
    before = [c.copy() for c in heights]
    fixed = [unaligned(np.zeros((h, w), np.uint16)) for _ in range(9)]
    assert gen.erode(heights, fixed, np.zeros(0, np.float32)) == 0.0
    for a, b, f in zip(heights, before, fixed):
        assert np.array_equal(a, b) and np.array_equal(f, oracle.format(b))
