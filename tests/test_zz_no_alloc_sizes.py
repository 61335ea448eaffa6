"""One first call of sol_gpu_batch_forward_adjoint_noalloc is enough for calls of every size.

The fused kernel has two builds, picked by the size of the call.  In a process
of its own (no other test has loaded either), after one call with no views at
all, small and large calls must leave the device's free memory as it is, and
calls whose first use is under stream capture must give the results of plain
ones."""
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parent.parent

SCRIPT = r"""
import ctypes as C
import sys
import torch
sys.path.insert(0, "tests")
from sol_b200 import capi, scenes
from sol_b200.renderer import GpuScene
from test_zz_no_alloc import _adjoint_views, _buffers

scene = scenes.cornell_box(0, textured=True, tex_size=32)
gs = GpuScene(scene)
cfg = scenes.CORNELL_CONFIG.to_c()
one = (capi.ScenePtr * 1)(gs.handle)
count = gs.param_layout()[0]
calls, targets = {}, {}
for name, (w, h, spp) in {"small": (24, 16, 2), "large": (131, 128, 12)}.items():   # either side of 94,720 paths
    views = [(0, scene.camera, w, h, 5, spp)]
    targets[name] = [torch.full((3, h, w), 0.25, device="cuda")]
    out = [_buffers(torch, views, [count]) for _ in range(2)]   # plain, captured
    calls[name] = [(f, g, l, _adjoint_views(capi, views, f, targets[name], g, l)) for f, g, l in out]
stream = torch.cuda.Stream()

def call(arr, n=1):
    capi.check(capi.lib.sol_gpu_batch_forward_adjoint_noalloc(one, 1, C.byref(cfg), arr, n, stream.cuda_stream), "call")

graphs = {name: torch.cuda.CUDAGraph() for name in calls}
torch.cuda.synchronize()
call(None, 0)   # the first call
torch.cuda.synchronize()
free = [torch.cuda.mem_get_info()[0]]
for name in ("small", "large", "small", "large"):
    f, g, l, arr = calls[name][0]
    for t in (*f, *g, l):
        t.zero_()
    torch.cuda.synchronize()
    call(arr)
    torch.cuda.synchronize()
    free.append(torch.cuda.mem_get_info()[0])
assert len(set(free)) == 1, free
for name in calls:
    f, g, l, arr = calls[name][1]
    with torch.cuda.graph(graphs[name], stream=stream, capture_error_mode="thread_local"):
        call(arr)
    graphs[name].replay()
    torch.cuda.synchronize()
    f0, g0, l0, _ = calls[name][0]
    assert f0[0].any() and torch.equal(f[0], f0[0])
    assert torch.allclose(l, l0, rtol=1e-9, atol=0.0)
    assert torch.allclose(g[0], g0[0], rtol=1e-4, atol=1e-4 * float(g0[0].abs().max()))
print("ok")
"""


def test_first_call_serves_every_size(built):
    r = subprocess.run([sys.executable, "-c", SCRIPT], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stdout[-500:] + r.stderr[-2000:]
