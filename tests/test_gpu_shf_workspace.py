"""The filter in a workspace that begins at any word of four bytes: every path, bit for bit as the
oracle; the paths that read words of eight are taken where the workspace is aligned to them.  An
address inside a word is refused before a launch."""
import ctypes as C

import numpy as np
import pytest

from test_gpu_shf import assert_same
from test_gpu_shf_fast import unpack
from test_gpu_shf_panels import sample_map

CASES = [((40, 37), 4, 5, "noise", 2), ((300, 41), 6, 80, "fields", 0), ((60, 33), 4, 40, "noise", 0)]


@pytest.mark.gpu
@pytest.mark.parametrize("path", [0, 1, 3])
@pytest.mark.parametrize("offset", [4, 8, 12, 16, 24, 40])
@pytest.mark.parametrize("ms,r,k,kind,taken", CASES, ids=["few", "panels", "many"])
def test_any_word(dev, oracle, shf_path, ms, r, k, kind, taken, offset, path):
    import torch
    shf_path(path)
    nn = (3, 3)
    sm = np.ascontiguousarray(sample_map(np.random.default_rng(k), ms, nn, k, kind))
    rc, off_ref, bins_ref = oracle.shf(sm, ms, nn, r)
    assert rc == 0
    size = dev.shf_workspace(ms, nn, r).numel()
    workspace = torch.full((size + 256,), 0x5A, dtype=torch.uint8, device="cuda")[offset:offset + size]
    assert workspace.data_ptr() % 16 == offset % 16
    off, bins, status = dev.shf_filter(torch.from_numpy(sm.view(np.int16)).cuda(), ms, nn, r, workspace=workspace)
    dev.status_check(status)
    assert_same(unpack(off, bins), (off_ref, bins_ref["Item"], bins_ref["Weight"]))
    if path == 0:
        assert dev.shf_filter_path(workspace, ms, nn, r) == (taken if offset % 8 == 0 else 0)


def test_an_address_inside_a_word_is_refused(stpgb):
    info = stpgb.NNInfo.make((64, 64), (3, 3))
    size = C.c_size_t(0)
    stpgb.check(stpgb.lib().stpgb_shf_workspace_size(C.byref(info), 4, 8, C.byref(size)))
    fake = C.c_void_p(0x1000)
    for at in (0x1001, 0x1002, 0x1007):
        rc = stpgb.lib().stpgb_shf_filter(fake, C.byref(info), 4, 8, C.c_void_p(at), size, fake, fake, 8, fake, None)
        assert rc == stpgb._capi.STPGB_EINVAL
        assert b"aligned" in stpgb.lib().stpgb_last_error()
