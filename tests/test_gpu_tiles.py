"""Camera rays of frames of at least 2^22 paths start at their tile's start nodes
(beam.cuh).  omv_render_device_static traces every ray from the scene's root:
the films of scenes without point lights are bit-identical."""
import ctypes as C
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch(gpu):
    return pytest.importorskip("torch")


def _both(gpu, torch, rs, cam, prm):
    H, W = cam.height, cam.width
    films = []
    st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    for static in (False, True):
        s = torch.zeros((H, W, 3), dtype=torch.float64, device="cuda")
        c = torch.zeros((H, W), dtype=torch.int32, device="cuda")
        args = [rs.handle, C.byref(cam), C.byref(prm), C.c_void_p(s.data_ptr()), None, C.c_void_p(c.data_ptr()), st]
        if static:
            gpu.check(gpu.lib().omv_render_device_static(*args))
        else:
            gpu.check(gpu.lib().omv_render_device(*args, None))
        films.append(s)
    torch.cuda.synchronize()
    return films


def _transformed(sc, M):
    M = np.asarray(M, dtype=np.float64)
    insts = [dataclasses.replace(i, transform=(M @ i.transform.astype(np.float64)).astype(np.float32)) for i in sc.instances]
    return dataclasses.replace(sc, instances=insts)


@pytest.fixture(scope="module")
def clutter(scenes):
    return scenes.scene_c2(64, 64, 1, tri_scale=0.03, sky_size=(128, 64), seed=5)


@pytest.mark.parametrize("view", range(12))
def test_film_equals_tracing_from_the_root(gpu, scenes, torch, clutter, view):
    """Views from inside the cloud of objects, from within an object's bounds and from far away, along and off the
    axes, with narrow and wide fields of view, at odd sizes and 1 to 470 samples per pixel (tiles of 1 to 512 pixels), of scenes scaled and sheared."""
    rng = np.random.default_rng(view)
    M = np.eye(4)
    if view % 3 == 1:
        M[:3, :3] *= [1e-3, 1.0, 1e3][(view // 3) % 3]
    if view % 3 == 2:
        M[:3, :3] = np.diag(rng.uniform(0.2, 3.0, 3)) @ (np.eye(3) + 0.4 * rng.normal(size=(3, 3)))
    sc = _transformed(clutter, M)
    scale = float(np.cbrt(abs(np.linalg.det(M[:3, :3]))))
    w, h, spp = [(1025, 513, 8), (2051, 2049, 1), (333, 41, 310), (511, 257, 33), (129, 70, 470), (1537, 700, 4)][view % 6]
    pos = np.zeros(3) if view % 4 == 0 else rng.uniform(-15, 15, 3) * scale
    if view % 4 == 3:
        pos = M[:3, :3] @ clutter.instances[view].transform[:3, 3].astype(np.float64)
    if view == 6:
        pos = np.array([0.0, 0.0, 300.0]) * scale
    fwd = rng.normal(size=3) if view % 4 and view != 6 else np.array([0.0, 0.0, -1.0])
    fwd /= np.linalg.norm(fwd)
    cam = gpu.PinholeCamera(w, h, tuple(pos), tuple(fwd), up=(0.0, 1.0, 0.0))
    cam.adjust_to_resolution()
    cam.set_y_fov([60.0, 3.0, 150.0][view % 3])
    rs = gpu.RenderScene(sc)
    a, b = _both(gpu, torch, rs, cam.to_c(), gpu.RendererParameters.for_scene(sc, samplesPerPixel=spp, seed=view).to_c())
    # (from inside a closed object the film is black on both sides)
    assert torch.equal(a, b) and (float(b.abs().max()) > 0 or view % 4 == 3)


def test_focus_zero_and_skewed_cameras(gpu, scenes, torch, clutter):
    """A camera without a beam (focus 0) and a view matrix that is not a rotation."""
    rs = gpu.RenderScene(clutter)
    prm = gpu.RendererParameters.for_scene(clutter, samplesPerPixel=16, seed=1).to_c()
    cam = gpu.PinholeCamera(970, 271)
    cam.adjust_to_resolution()
    a, b = _both(gpu, torch, rs, cam.to_c(), prm)
    assert torch.equal(a, b)
    cam.set_y_fov(70.0)
    cam.rotation = np.array([[1.3, 0.2, 0.1], [-0.3, 0.7, 0.2], [0.1, -0.4, 2.0]], dtype=np.float32)
    a, b = _both(gpu, torch, rs, cam.to_c(), prm)
    assert torch.equal(a, b)


def test_many_instances_and_masked_materials(gpu, scenes, torch, clutter):
    """More instances in a tile than a list holds, and hits that are skipped."""
    rng = np.random.default_rng(3)
    insts = []
    for k in range(1500):
        T = np.eye(4)
        T[:3, :3] = scenes.random_rotation(rng) * 0.3
        T[:3, 3] = rng.uniform(-3, 3, 3) + [0, 0, -12]
        insts.append(scenes.Instance(T.astype(np.float32), int(rng.integers(0, 64))))
    mats = [dataclasses.replace(m, alpha_mode=2, base_color=m.base_color[:3] + (0.0,)) if i % 2 else m
            for i, m in enumerate(clutter.materials)]
    sc = dataclasses.replace(clutter, instances=insts, materials=mats)
    cam = gpu.PinholeCamera(801, 601)
    cam.adjust_to_resolution()
    cam.set_y_fov(40.0)
    rs = gpu.RenderScene(sc)
    a, b = _both(gpu, torch, rs, cam.to_c(), gpu.RendererParameters.for_scene(sc, samplesPerPixel=9, seed=2).to_c())
    assert torch.equal(a, b)


@pytest.mark.parametrize("size", [(1537, 700, 4), (333, 41, 310), (1, 70_001, 60), (70_001, 1, 61)])
def test_lists_of_several_waves(gpu, torch, clutter, size):
    """Waves that begin and end inside tile rows and pixels, with all lists of the frame made at once (a handle's first
    frame has the room for them) and with those of each wave's tiles (a handle whose scratch was made for another
    frame, too small a wave for its tiles included)."""
    w, h, spp = size
    cam = gpu.PinholeCamera(w, h)
    cam.position = np.array([0.5, 1.0, 12.0])
    cam.adjust_to_resolution()
    cam.set_y_fov(60.0)
    first, used = gpu.RenderScene(clutter), gpu.RenderScene(clutter)
    small = gpu.PinholeCamera(1100, 1000).to_c()
    _both(gpu, torch, used, small, gpu.RendererParameters.for_scene(clutter, samplesPerPixel=1).to_c())
    want = None
    for wave in (0, 1_000_003, 70_001, 999):
        if wave == 999 and w > 1:
            continue
        prm = gpu.RendererParameters.for_scene(clutter, samplesPerPixel=spp, seed=8, wave_paths=wave).to_c()
        for rs in (used, first):
            s = torch.zeros((h, w, 3), dtype=torch.float64, device="cuda")
            c = torch.zeros((h, w), dtype=torch.int32, device="cuda")
            if wave == 0:
                if rs is first:
                    continue
                gpu.check(gpu.lib().omv_render_device_static(rs.handle, C.byref(cam.to_c()), C.byref(prm), C.c_void_p(s.data_ptr()),
                                                             None, C.c_void_p(c.data_ptr()), None))
                want = s
            else:
                gpu.check(gpu.lib().omv_render_device(rs.handle, C.byref(cam.to_c()), C.byref(prm), C.c_void_p(s.data_ptr()), None,
                                                      C.c_void_p(c.data_ptr()), None, None))
            torch.cuda.synchronize()
            assert int(c.min()) == int(c.max()) == spp
            assert float((s - want).abs().max()) <= 1e-9 * float(want.abs().max())
