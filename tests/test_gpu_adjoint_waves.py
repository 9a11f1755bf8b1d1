"""The replay's wave loop: several waves, many jobs, pixels without a
derivative, other streams and graph capture.  A gradient is a sum of a few
million FP32 terms of either sign per material slot, kept in FP64 from block
to block: orders of summation agree to 1e-4 of the largest component."""
import ctypes as C
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
RTOL = 1e-4


def _close(a, b):
    scale = float(b.abs().max())
    assert scale > 0
    assert float((a - b).abs().max()) <= RTOL * scale


class Scene:
    def __init__(self, gpu, scenes, torch, side, **kw):
        self.gpu, self.torch = gpu, torch
        self.sc = scenes.scene_materials(side, side, 1, **{"tris": 4_000, "n_materials": 4, "bounces": 4, "seed": 3, **kw})
        self.rs = gpu.RenderScene(self.sc)
        self.cam = gpu.PinholeCamera.from_spec(self.sc.camera).to_c()
        g = torch.Generator(device="cuda").manual_seed(5)
        self.adj = torch.rand((side, side, 3), device="cuda", generator=g) - 0.3

    def params(self, spp, offset=0, seed=11, **kw):
        return self.gpu.RendererParameters.for_scene(self.sc, samplesPerPixel=spp, sample_offset=offset, seed=seed, **kw).to_c()

    def grad(self, spp, adj=None, stream=None, out=None, **kw):
        adj = self.adj if adj is None else adj
        g = self.torch.zeros((len(self.sc.materials), 11), device="cuda") if out is None else out
        st = stream if stream is not None else self.torch.cuda.current_stream()
        self.gpu.check(self.gpu.lib().omv_adjoint(self.rs.handle, C.byref(self.cam), C.byref(self.params(spp, **kw)),
                                                  C.c_void_p(adj.data_ptr()), C.c_void_p(g.data_ptr()),
                                                  C.c_void_p(st.cuda_stream)))
        return g


@pytest.fixture(scope="module")
def torch(gpu):
    return pytest.importorskip("torch")


def test_several_waves_sum_their_sample_ranges(gpu, scenes, torch):
    """256x256 at 208 samples do not fit one wave's records: the gradient is the mean of the ranges' gradients."""
    s = Scene(gpu, scenes, torch, 256)
    whole = s.grad(208)
    parts = [s.grad(52, offset=52 * k) for k in range(4)]
    torch.cuda.synchronize()
    _close(whole, sum(p.double() for p in parts) / 4)


@pytest.mark.parametrize("side,spp", [(1, 1), (3, 5), (33, 3)])
def test_pixels_without_a_derivative_add_nothing(gpu, scenes, torch, side, spp):
    s = Scene(gpu, scenes, torch, side)
    assert float(s.grad(spp, adj=torch.zeros_like(s.adj)).abs().max()) == 0.0
    mask = (torch.arange(side * side, device="cuda").reshape(side, side, 1) % 3 == 0).float()
    a = s.grad(spp * 16, adj=s.adj * mask)
    b = s.grad(spp * 16, adj=s.adj * (1 - mask)) if side > 1 else torch.zeros_like(a)
    whole = s.grad(spp * 16)
    torch.cuda.synchronize()
    _close(a + b, whole)


@pytest.mark.parametrize("light_bounces,camera_bounces,max_len", [(0, 3, 8), (3, 1, 8), (15, 15, 30), (2, 4, 1)])
def test_bounce_limits_accumulate_into_the_buffer(gpu, scenes, torch, light_bounces, camera_bounces, max_len):
    """The gradient is added to what the buffer holds, at every bounce limit."""
    s = Scene(gpu, scenes, torch, 24, sky=True)
    kw = {"lightBouncesN": light_bounces, "cameraBouncesN": camera_bounces, "maxPathLength": max_len}
    once = s.grad(64, **kw)
    twice = s.grad(64, out=once.clone(), **kw)
    torch.cuda.synchronize()
    _close(twice, 2 * once)


def test_many_jobs_of_uneven_size_match_single_calls(gpu, scenes, torch):
    """30 jobs of 4 and 8 materials (more gradient sums than one sequence of waves holds) with material sets of their
    own; two jobs share a buffer."""
    parts = [scenes.scene_materials(8, 8, 1, tris=3_000, n_materials=4 + 4 * (p % 2), seed=p, bounces=3) for p in range(5)]
    group = gpu.RenderScene.group(parts)
    br = gpu.BatchRenderer(group, gpu.RendererParameters.for_scene(parts[0]))
    alone = [gpu.RenderScene(sc) for sc in parts]
    rng = np.random.default_rng(1)
    film = (torch.zeros(1, device="cuda"), None, torch.zeros(1, device="cuda"))
    jobs, adjs, grads, want = [], [], [], []
    for j in range(30):
        p = j % len(parts)
        cam = gpu.PinholeCamera.from_spec(parts[p].camera)
        cam.width, cam.height = int(rng.integers(1, 40)), int(rng.integers(1, 40))
        cam.adjust_to_resolution()
        cam.set_y_fov(45.0)
        spp = int(rng.integers(1, 40))
        a = torch.tensor(rng.uniform(-1, 1, (cam.height, cam.width, 3)), dtype=torch.float32, device="cuda")
        w = torch.zeros((len(parts[p].materials), 11), device="cuda")
        prm = gpu.RendererParameters.for_scene(parts[0], samplesPerPixel=spp, seed=j, sample_offset=j).to_c()
        gpu.check(gpu.lib().omv_adjoint(alone[p].handle, C.byref(cam.to_c()), C.byref(prm), C.c_void_p(a.data_ptr()),
                                        C.c_void_p(w.data_ptr()), C.c_void_p(torch.cuda.current_stream().cuda_stream)))
        jobs.append(br.job(cam, spp, film, seed=j, sample_offset=j, part=p))
        adjs.append(a)
        grads.append(torch.zeros_like(w))
        want.append(w)
    grads[5] = grads[0]  # the same scene (part 0)
    want[0] += want[5]
    br.adjoint(jobs, adjs, grads)
    torch.cuda.synchronize()
    for j in (i for i in range(30) if i != 5):
        if float(want[j].abs().max()) > 0:
            _close(grads[j], want[j])
        else:
            assert float(grads[j].abs().max()) == 0.0


def test_two_streams_share_the_records(gpu, scenes, torch):
    s = Scene(gpu, scenes, torch, 96)
    want = s.grad(64)
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    outs = [torch.zeros_like(want) for _ in range(8)]
    torch.cuda.synchronize()
    for i, g in enumerate(outs):
        s.grad(64, stream=streams[i % 2], out=g)
    torch.cuda.synchronize()
    for g in outs:
        _close(g, want)


def test_capture_into_a_graph(gpu, scenes, torch):
    """A captured replay has its own records: it repeats while direct calls run in between."""
    s = Scene(gpu, scenes, torch, 48)
    want = s.grad(32)
    torch.cuda.synchronize()
    out = torch.zeros_like(want)
    graph = torch.cuda.CUDAGraph()
    stream = torch.cuda.Stream()
    with torch.cuda.graph(graph, stream=stream, capture_error_mode="relaxed"):
        s.grad(32, stream=torch.cuda.current_stream(), out=out)
    for _ in range(3):
        graph.replay()
        s.grad(64)
    torch.cuda.synchronize()
    _close(out, 3 * want)
