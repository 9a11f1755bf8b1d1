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


def test_handles_on_threads_of_their_own(gpu, scenes):
    """Four threads, each with a handle and a stream: gradients of two sizes and ray queries of two, all at once, are those
    of calls one after another."""
    import ctypes as C
    import threading

    import numpy as np

    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(2)
    rays = np.zeros((40_000, 8), np.float32)
    rays[:, 0:3], rays[:, 4:7], rays[:, 7] = rng.uniform(-2, 2, (len(rays), 3)) + [0, 0, 6], rng.normal(size=(len(rays), 3)), 3e38
    work = []
    for k in range(4):
        sc = scenes.scene_materials(64, 64, 1, tris=4_000, n_materials=4, bounces=4, seed=k)
        w = {"sc": sc, "rs": gpu.RenderScene(sc), "stream": torch.cuda.Stream(), "cam": gpu.PinholeCamera.from_spec(sc.camera).to_c(),
             "adj": torch.rand((64, 64, 3), device="cuda", generator=torch.Generator(device="cuda").manual_seed(k)) - 0.3}
        w["prm"] = [gpu.RendererParameters.for_scene(sc, seed=k, samplesPerPixel=spp).to_c() for spp in (16, 48)]
        work.append(w)

    def grad(w, i, out):
        gpu.check(gpu.lib().omv_adjoint(w["rs"].handle, C.byref(w["cam"]), C.byref(w["prm"][i]), C.c_void_p(w["adj"].data_ptr()),
                                        C.c_void_p(out.data_ptr()), C.c_void_p(w["stream"].cuda_stream)))

    new = lambda w: torch.zeros((len(w["sc"].materials), 11), device="cuda")
    want = [[new(w), new(w)] for w in work]
    outs = [[new(w), new(w)] for w in work]
    torch.cuda.synchronize()
    hits = []
    for w, g in zip(work, want):
        for i in (0, 1):
            grad(w, i, g[i])
        torch.cuda.synchronize()
        hits.append([w["rs"].trace(rays[:n]) for n in (3_000, 40_000)])
    errors = []

    def run(k):
        try:
            torch.cuda.set_device(0)
            for step in range(12):
                i = (step + k) % 2
                grad(work[k], i, outs[k][i])
                got = work[k]["rs"].trace(rays[:(3_000, 40_000)[1 - i]])
                if not np.array_equal(got.view(np.uint32), hits[k][1 - i].view(np.uint32)):
                    errors.append((k, step))
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=run, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not errors, errors
    for g, w in zip(outs, want):
        for a, b in zip(g, w):
            scale = float(b.abs().max())
            assert scale > 0 and float((a - 6 * b).abs().max()) <= 1e-4 * 6 * scale
