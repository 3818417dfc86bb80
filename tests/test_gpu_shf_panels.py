"""The filter's row bands where a row is cut into panels and a panel has a palette of its own: chunks
of more than 8 values, chunks wider than one panel, and the ones next to them that take the general
slides, against the oracle: offsets, items, weights and bin order bit-exact."""
import zlib

import numpy as np
import pytest

from test_gpu_shf import assert_same
from test_gpu_shf_fast import run, unpack

pytestmark = pytest.mark.gpu


def sample_map(rng, ms, nn, k, kind):
    """A sample map of values spread over the 16-bit range, 0 and 65535 included: `noise` of k values,
    `fields` of k by k pixels with a value each (the same ones come again further away), `specks`
    of k values on one, `stripes` of k columns."""
    h, w = ms[1] * nn[1], ms[0] * nn[0]
    values = np.concatenate([[0, 65535], rng.choice(np.arange(1, 65535), 60, replace=False)]).astype(np.uint16)
    if kind == "noise":
        return rng.permutation(values[:k])[rng.integers(0, k, (h, w))]
    y, x = np.mgrid[0:h, 0:w]
    if kind == "fields":
        return values[((x // k) * 7 + (y // k) * 11) % 62]
    if kind == "stripes":
        return values[(x // k) % 62]
    speck = rng.random((h, w)) < 0.002
    return np.where(speck, values[rng.integers(0, k, (h, w))], values[1]).astype(np.uint16)


CASES = [
    # name, map size, nn, radius, k, kind
    ("nine", (40, 40), (3, 3), 4, 9, "noise"),
    ("sixteen-odd", (37, 29), (3, 3), 4, 16, "noise"),
    ("seventeen", (37, 29), (3, 3), 4, 17, "noise"),
    ("one-row", (64, 1), (3, 33), 16, 12, "noise"),
    ("one-column", (1, 64), (33, 3), 16, 12, "noise"),
    ("one-pixel", (1, 1), (9, 9), 4, 10, "noise"),
    ("many-by-band", (300, 211), (3, 3), 6, 80, "fields"),
    ("one-panel-full", (1000, 13), (3, 9), 12, 11, "specks"),
    ("one-panel-and-a-column", (1001, 13), (3, 9), 12, 11, "specks"),
    ("panel-edges", (1999, 9), (3, 9), 12, 16, "noise"),
    ("panel-edges-few", (2000, 9), (3, 9), 12, 5, "noise"),
    ("fields-many-panels", (3100, 21), (3, 5), 20, 210, "fields"),
    ("stripes-many-panels", (4500, 10), (3, 9), 10, 150, "stripes"),
    ("beyond-one-palette", (4300, 7), (3, 9), 4, 8, "noise"),
    ("widest-radius", (800, 12), (3, 31), 126, 13, "specks"),
    ("past-widest-radius", (260, 12), (3, 31), 128, 13, "specks"),
    ("crowded-in-one-panel", (2100, 8), (3, 9), 8, 62, "specks"),
]


@pytest.mark.parametrize("path", [0, 3])
@pytest.mark.parametrize("name,ms,nn,r,k,kind", CASES, ids=[c[0] for c in CASES])
def test_panels_vs_oracle(dev, oracle, shf_path, path, name, ms, nn, r, k, kind):
    shf_path(path)
    rng = np.random.default_rng(zlib.crc32(name.encode()))
    sm = np.ascontiguousarray(sample_map(rng, ms, nn, k, kind))
    rc, off_ref, b = oracle.shf(sm, ms, nn, r)
    assert rc == 0
    off, bins, status, _ = run(dev, sm, ms, nn, r)
    dev.status_check(status)
    assert_same(unpack(off, bins), (off_ref, b["Item"], b["Weight"]), name)


def test_panels_repeated_calls_same_workspace(dev, oracle, shf_path):
    """A crowded chunk, one of few values, one with a palette per panel and the crowded one again
    through one workspace."""
    import torch
    shf_path(0)
    rng = np.random.default_rng(21)
    ms, r = (120, 70), 8
    maps = [sample_map(rng, ms, (3, 3), k, kind) for k, kind in ((40, "noise"), (4, "noise"), (60, "fields"))]
    ws = dev.shf_workspace(ms, (3, 3), r)
    for n, sm in enumerate(maps + maps[:1]):
        rc, off_ref, b = oracle.shf(np.ascontiguousarray(sm), ms, (3, 3), r)
        t = torch.from_numpy(np.ascontiguousarray(sm).view(np.int16)).cuda()
        off, bins, status = dev.shf_filter(t, ms, (3, 3), r, workspace=ws)
        dev.status_check(status)
        assert_same(unpack(off, bins), (off_ref, b["Item"], b["Weight"]), n)


def test_panels_refuse_what_the_slides_refuse(stpgb, dev, oracle, shf_path):
    """max_items below what a window holds is a capacity error however the chunk is filtered: 12
    values with 11 allowed, and one column whose window and the row it still holds have 10 of the
    allowed 9, though each window has 9."""
    shf_path(0)
    rng = np.random.default_rng(5)
    sm = sample_map(rng, (40, 30), (3, 3), 12, "noise")
    off, bins, status, _ = run(dev, sm, (40, 30), (3, 3), 6, max_items=11)
    with pytest.raises(stpgb.STPCapacityError):
        dev.status_check(status)
    rows = np.arange(3 * 40) % 10
    sm = np.ascontiguousarray(np.repeat(rows[:, None], 3 * 40, 1).astype(np.uint16))
    results = []
    for path in (0, 3):
        shf_path(path)
        off, bins, status, _ = run(dev, sm, (40, 40), (3, 3), 4, max_items=9)
        try:
            dev.status_check(status)
            results.append("taken")
        except stpgb.STPCapacityError:
            results.append("refused")
    assert results[0] == results[1] == "refused"


def test_panels_short_bins_capacity(stpgb, dev, oracle, shf_path):
    """A bins capacity 5 short of the total: ECAPACITY on the status, every offset still written
    and the bins that fit equal to the oracle's."""
    shf_path(0)
    rng = np.random.default_rng(9)
    ms, r = (1300, 12), 10
    sm = np.ascontiguousarray(sample_map(rng, ms, (3, 3), 14, "specks"))
    rc, off_ref, b = oracle.shf(sm, ms, (3, 3), r)
    total = int(off_ref[-1])
    off, bins, status, _ = run(dev, sm, ms, (3, 3), r, cap=total - 5)
    with pytest.raises(stpgb.STPCapacityError):
        dev.status_check(status)
    got_off, items, weights = unpack(off, bins, total - 5)
    assert np.array_equal(got_off, off_ref)
    assert np.array_equal(items, b["Item"][:total - 5])
    assert np.array_equal(weights.view(np.uint32), b["Weight"][:total - 5].view(np.uint32))
