"""shiro_gpu_render_static moves no device memory whatever the process rendered
before: nothing, or a frame small enough for another launch shape of the plain
form than the one that follows.  A process of its own each: the driver keeps the
thread-local memory that earlier kernels of a process needed."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CHILD = r"""
import ctypes as C, sys
import torch
from shiro_gb300 import GpuBackend, RenderSettings, scenes
from shiro_gb300.abi import Aovs, render_desc

ext, warm = sys.argv[1] == "ext", int(sys.argv[2])
torch.cuda.init()
gpu = GpuBackend(0)
lib = gpu.lib
lib.shiro_gpu_render_static.argtypes = [C.c_void_p] * 4
lib.shiro_gpu_render_static.restype = C.c_int
w = scenes.sphere_workload(512, 512, 4, 8, env_width=128, env_height=64)
if ext:
    w.scene.materials[0].opacity = 0.5
gpu.upload_scene(w.scene)
if warm:
    st = RenderSettings(width=warm, height=warm, samples_per_pixel=1, max_depth=8, diffuse_depth=8, specular_depth=8,
                        backend=1)
    gpu.render(w.scene, w.camera, st)
planes = [torch.zeros(512 * 512 * c, device="cuda") for c in (4, 3, 3, 1)]
aov = Aovs(*[C.cast(C.c_void_p(p.data_ptr()), C.POINTER(C.c_float)) for p in planes], 1, 0)
torch.cuda.synchronize()
before = torch.cuda.mem_get_info()[0]
req = render_desc(w.camera, w.settings, 0, 4)
assert lib.shiro_gpu_render_static(gpu.handle, C.byref(req), None, C.byref(aov)) == 0
torch.cuda.synchronize()
print("moved", before - torch.cuda.mem_get_info()[0])
"""


@pytest.mark.parametrize("warm", [0, 32])
@pytest.mark.parametrize("kind", ["lean", "ext"])
def test_no_memory_moves_after_any_warm_up(kind, warm):
    pytest.importorskip("torch")
    r = subprocess.run([sys.executable, "-c", CHILD, kind, str(warm)], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    assert r.stdout.split()[-2:] == ["moved", "0"], r.stdout
