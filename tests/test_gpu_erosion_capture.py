"""Erosion in tiles on one stream while another one is captured: the capture goes on, whatever its mode,
and the call erodes the map.  A process of its own, so that the tiles' pool is made meanwhile."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = """
import ctypes as C, sys
import torch
sys.path[:0] = [{root!r}, {tests!r}]
import helpers
import superterrainplus_gb300 as stpgb
from test_gpu_erosion import terrain
n, drops = 300, 200
before = torch.from_numpy(terrain(n, n, 1)).cuda()
maps = [before.clone() for _ in range(3)]
starts = torch.rand(2 * drops, device="cuda") * 200 + 50
idx, w = (torch.from_numpy(a).cuda() for a in stpgb.erosion_brush(n, 3))
info, rain = stpgb.NNInfo.make((n, n), (1, 1)), stpgb.RaindropSetting(**helpers.raindrop_dict(drops, radius=3, lifetime=20))
ptr = lambda t: C.c_void_p(t.data_ptr())
x = torch.zeros(8, device="cuda")
side = torch.cuda.Stream()
torch.cuda.synchronize()
for m in maps:
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, capture_error_mode={mode!r}):
        x.add_(1)
        stpgb.check(stpgb.lib().stpgb_hydraulic_erosion_ex(ptr(m), C.byref(info), C.byref(rain), ptr(starts), drops,
                                                           ptr(idx), ptr(w), idx.numel(), None, None, 0, 1, 4,
                                                           C.c_void_p(side.cuda_stream)))
        x.add_(1)
    graph.replay()
    torch.cuda.synchronize()
    assert not torch.equal(m, before)
assert x[0].item() == 6.0
print("fine")
"""


@pytest.mark.parametrize("mode", ["global", "thread_local", "relaxed"])
def test_tiles_beside_a_capture(mode):
    program = PROGRAM.format(root=ROOT, tests=os.path.join(ROOT, "tests"), mode=mode)
    r = subprocess.run([sys.executable, "-c", program], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "fine" in r.stdout, r.stderr[-2000:]
