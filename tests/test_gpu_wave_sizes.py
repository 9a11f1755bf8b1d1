"""One handle of a scene with point lights renders frames and batches of mixed
sizes: small waves (light subpaths beside the camera rays), waves above 2^22
paths, and a short last wave of a large frame or batch after a small frame.
The films are those of a fresh handle up to the order of the FP32 additions to
a path's radiance (at most 42 terms of half an ulp: 5e-6)."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu
RTOL = 5e-6


@pytest.fixture(scope="module")
def torch(gpu):
    return pytest.importorskip("torch")


def _film(torch, w, h):
    return torch.zeros((h, w, 3), dtype=torch.float64, device="cuda"), None, torch.zeros((h, w), dtype=torch.int32, device="cuda")


def _frame(gpu, scenes, torch, rs, w, h, spp, wave_paths=0):
    sc = scenes.scene_c1(w, h, spp)
    cam = gpu.PinholeCamera.from_spec(sc.camera).to_c()
    prm = gpu.RendererParameters.for_scene(sc, seed=7, wave_paths=wave_paths).to_c()
    s, _, c = _film(torch, w, h)
    gpu.check(gpu.lib().omv_render_device(rs.handle, C.byref(cam), C.byref(prm), C.c_void_p(s.data_ptr()), None,
                                          C.c_void_p(c.data_ptr()), C.c_void_p(torch.cuda.current_stream().cuda_stream), None))
    torch.cuda.synchronize()
    assert int(c.min()) == int(c.max()) == spp
    return s


def _close(a, b):
    assert float((a - b).abs().max()) <= RTOL * float(b.abs().max())


# width, height, samples, wave_paths (0: as large as fits)
ORDERS = {
    "small, then a short last wave above 2^22": [(64, 64, 1, 0), (512, 512, 20, (1 << 22) + 37)],
    "growing": [(9, 7, 3, 0), (120, 90, 16, 0), (512, 512, 20, (1 << 22) + 5)],
    "mixed": [(512, 512, 20, 5_000_001), (9, 7, 3, 0), (1024, 512, 16, (1 << 22) + 1), (120, 90, 16, 0), (9, 7, 3, 50),
              (300, 200, 20, 999_983)],
}


@pytest.mark.parametrize("order", ORDERS, ids=lambda k: k.replace(" ", "-"))
def test_frames_of_mixed_sizes_on_one_handle(gpu, scenes, torch, order):
    rs = gpu.RenderScene(scenes.scene_c1(8, 8, 1))
    got = [_frame(gpu, scenes, torch, rs, *f) for f in ORDERS[order]]
    for f, a in zip(ORDERS[order], got):
        _close(a, _frame(gpu, scenes, torch, gpu.RenderScene(scenes.scene_c1(8, 8, 1)), *f))


@pytest.mark.parametrize("graph", [False, True])
def test_batch_with_a_short_last_wave_after_a_preview(gpu, scenes, torch, graph):
    """50.3M paths do not fit one wave's scratch (32 GiB, about 712 bytes per path)."""
    sc = scenes.scene_c1(1024, 1024, 24)

    def batch(rs):
        br = gpu.BatchRenderer(rs, gpu.RendererParameters.for_scene(sc))
        cam = gpu.PinholeCamera.from_spec(sc.camera)
        films = [_film(torch, 1024, 1024) for _ in range(2)]
        jobs = [br.job(cam, 24, f, seed=k) for k, f in enumerate(films)]
        br.render(jobs, graph=graph)
        torch.cuda.synchronize()
        assert all(int(f[2].min()) == int(f[2].max()) == 24 for f in films)
        return [f[0] for f in films]

    rs = gpu.RenderScene(sc)
    _frame(gpu, scenes, torch, rs, 64, 64, 1)
    got = batch(rs)
    _frame(gpu, scenes, torch, rs, 120, 90, 16)
    for a, b in zip(got, batch(gpu.RenderScene(sc))):
        _close(a, b)
