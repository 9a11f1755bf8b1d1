"""Memory that a gradient or a ray query needs besides the scene: shared by the
handles of a process, kept for the next call, given back with the last handle."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

_MANY_HANDLES = r"""
import ctypes as C, importlib, sys
sys.path.insert(0, sys.argv[1])
import numpy as np, torch
gpu = importlib.import_module("openmaterial-validation_gb300")
scenes = importlib.import_module("openmaterial-validation_gb300.scenes")
sc = scenes.scene_materials(128, 128, 1, tris=4_000, n_materials=4, bounces=4, seed=3)
cam, prm = gpu.PinholeCamera.from_spec(sc.camera).to_c(), gpu.RendererParameters.for_scene(sc, samplesPerPixel=64, seed=1).to_c()
adj = torch.rand((128, 128, 3), device="cuda")
rays = np.zeros((2_000_000, 8), np.float32)
rays[:, 2], rays[:, 6], rays[:, 7] = -1.0, -1.0, 3e38
grads = []

def use(handles):
    for k, rs in enumerate(handles):
        g = torch.zeros((len(sc.materials), 11), device="cuda")
        stream = torch.cuda.Stream() if k % 3 == 0 else torch.cuda.current_stream()
        torch.cuda.synchronize()
        gpu.check(gpu.lib().omv_adjoint(rs.handle, C.byref(cam), C.byref(prm), C.c_void_p(adj.data_ptr()), C.c_void_p(g.data_ptr()),
                                        C.c_void_p(stream.cuda_stream)))
        stream.synchronize()
        rs.trace(rays)
        grads.append(g)

handles = [gpu.RenderScene(sc) for _ in range(12)]
use(handles[:1])  # kernels and their local memory are loaded
torch.cuda.synchronize()
one = torch.cuda.mem_get_info()[0]
use(handles[1:])
torch.cuda.synchronize()
many = torch.cuda.mem_get_info()[0]
del handles
import gc
gc.collect()
torch.cuda.synchronize()
none = torch.cuda.mem_get_info()[0]
scale = float(grads[0].abs().max())
assert scale > 0 and all(float((g - grads[0]).abs().max()) <= 1e-4 * scale for g in grads)
print("RESULT", one - many, none - one)
"""


def test_many_handles_share_records_and_ray_buffers(gpu):
    """1.2 GB of records, 128 MB of rays and hits: eleven more handles, on streams of their own too, take next to nothing
    more, and with the last handle the memory is free again."""
    r = subprocess.run([sys.executable, "-c", _MANY_HANDLES, ROOT], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    more, back = (int(x) for x in r.stdout.split("RESULT")[1].split())
    assert more < 256 << 20, more
    assert back > 1 << 30, back


_SIZES = r"""
import importlib, sys
sys.path.insert(0, sys.argv[1])
import numpy as np, torch
gpu = importlib.import_module("openmaterial-validation_gb300")
scenes = importlib.import_module("openmaterial-validation_gb300.scenes")
rs = gpu.RenderScene(scenes.scene_mixed(8, 8, 1))
rng = np.random.default_rng(0)
rays = np.zeros((6_000_000, 8), np.float32)
rays[:, 0:3], rays[:, 4:7], rays[:, 7] = rng.uniform(-3, 3, (len(rays), 3)) + [0, 0, -8], rng.normal(size=(len(rays), 3)), 3e38
want = np.concatenate([rs.trace(rays[k:k + 500_000]) for k in range(0, len(rays), 500_000)])
torch.cuda.synchronize()
free0 = torch.cuda.mem_get_info()[0]
for n in (1, 6_000_000, 33_000, 1_000_003, 5_000_000, 7, 4_194_304, 4_194_305):  # kept up to 2^22 rays
    assert np.array_equal(rs.trace(rays[:n]).view(np.uint32), want[:n].view(np.uint32)), n
print("RESULT", free0 - torch.cuda.mem_get_info()[0])
"""


def test_ray_queries_of_mixed_sizes_keep_little(gpu):
    """Buffers above 256 MB are freed with their call, smaller ones are kept: 64 + 256 MB and less than as much again."""
    r = subprocess.run([sys.executable, "-c", _SIZES, ROOT], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    assert int(r.stdout.split("RESULT")[1]) < 640 << 20
