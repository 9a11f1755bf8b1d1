"""Connection rays run beside the next bounce's extension rays and the light
subpaths of small frames beside the camera's first hits, on a second stream;
omv_render_device_static runs one launch after another.  Films of lit scenes
agree up to the order of the FP32 additions to a path's radiance (at most 42
terms of half an ulp: 5e-6); MIS films of scenes without lights, where one
environment ray at a time reaches a path, are bit-identical to a one-by-one run."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


def _frames(gpu, torch, rs, cam, prm, static, n=1, stream=None):
    H, W = cam.height, cam.width
    st = stream if stream is not None else torch.cuda.current_stream()
    with torch.cuda.stream(st):
        s = torch.zeros((H, W, 3), dtype=torch.float64, device="cuda")
        c = torch.zeros((H, W), dtype=torch.int32, device="cuda")
        for _ in range(n):
            args = [rs.handle, C.byref(cam), C.byref(prm), C.c_void_p(s.data_ptr()), None, C.c_void_p(c.data_ptr()),
                    C.c_void_p(st.cuda_stream)]
            gpu.check(gpu.lib().omv_render_device_static(*args) if static else gpu.lib().omv_render_device(*args, None))
        out = s / n
    st.synchronize()
    assert int(c.min()) == int(c.max()) == n * prm.samples_per_pixel
    return out


@pytest.mark.parametrize("name", ["c1", "lights", "mixed", "textured"])
@pytest.mark.parametrize("size", [(9, 7, 3), (120, 90, 16)])
def test_lit_frames(gpu, scenes, name, size):
    torch = pytest.importorskip("torch")
    sc = getattr(scenes, f"scene_{name}")(*size)
    rs = gpu.RenderScene(sc)
    cam = gpu.PinholeCamera.from_spec(sc.camera).to_c()
    prm = gpu.RendererParameters.for_scene(sc, seed=4).to_c()
    want = _frames(gpu, torch, rs, cam, prm, True)
    for stream in (None, torch.cuda.Stream()):  # several frames back to back, nothing waited for in between
        got = _frames(gpu, torch, rs, cam, prm, False, n=5, stream=stream)
        assert float((got - want).abs().max()) <= 5e-6 * float(want.abs().max())


def test_mis_frames_and_their_kernels_timed_alone(gpu, scenes):
    torch = pytest.importorskip("torch")
    sc = scenes.scene_c2(120, 67, 16, tri_scale=0.03, sky_size=(128, 64))
    rs = gpu.RenderScene(sc)
    cam = gpu.PinholeCamera.from_spec(sc.camera).to_c()
    prm = gpu.RendererParameters.for_scene(sc, seed=4, estimator=1).to_c()
    a = _frames(gpu, torch, rs, cam, prm, False)
    prm.time_kernels = 1
    assert torch.equal(a, _frames(gpu, torch, rs, cam, prm, False))
