"""Queues of at most 2^15 rays are traced with eight lanes per ray, longer ones
with one ray per thread: the same frame in one wave (first bounces in long
queues) and in waves of a few hundred to a few thousand paths (every queue
short) has the same hits, so the film of a scene without point lights is
bit-identical, and with point lights equal up to the order of the FP32
additions to a path's radiance (at most 42 terms of half an ulp: 5e-6)."""
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _render(gpu, rs, sc, **kw):
    r = gpu.BDPTRenderer()
    r.set_scene(rs)
    r.set_parameters(gpu.RendererParameters.for_scene(sc, seed=9, **kw))
    _, s, _, c = r.render(gpu.PinholeCamera.from_spec(sc.camera), sums=True)
    assert r.last_stats["stack_overflows"] == 0
    return s, c


@pytest.mark.parametrize("estimator", [0, 1])
@pytest.mark.parametrize("waves", [32, 4096])
def test_unlit_film_does_not_depend_on_the_queue_length(gpu, scenes, estimator, waves):
    sc = scenes.scene_c2(96, 41, 32, tri_scale=0.05, sky_size=(128, 64))
    if waves < 4096:
        sc.camera.width, sc.camera.height, sc.render.samples_per_pixel = 7, 3, 32
    rs = gpu.RenderScene(sc)
    a, ca = _render(gpu, rs, sc, estimator=estimator)
    b, cb = _render(gpu, rs, sc, estimator=estimator, wave_paths=waves)
    assert np.array_equal(ca, cb) and np.array_equal(a, b)


@pytest.mark.parametrize("size", [(1024, 512, 64), (1023, 517, 65)])
def test_rays_grouped_over_several_shading_steps(gpu, scenes, size):
    """One wave of 2^25 paths or more groups its rays over windows of several steps, waves of 2^22 step by step."""
    sc = scenes.scene_c2(*size, tri_scale=0.02, sky_size=(128, 64))
    rs = gpu.RenderScene(sc)
    a, ca = _render(gpu, rs, sc)
    b, cb = _render(gpu, rs, sc, wave_paths=size[2] << 16)
    assert np.array_equal(ca, cb) and np.array_equal(a, b)


@pytest.mark.parametrize("name", ["c1", "mixed", "textured"])
def test_lit_film_does_not_depend_on_the_queue_length(gpu, scenes, name):
    """Conductors, transmission, blended and texture-masked materials (retries past masked hits)."""
    sc = getattr(scenes, f"scene_{name}")(80, 60, 32)
    rs = gpu.RenderScene(sc)
    a, ca = _render(gpu, rs, sc)
    b, cb = _render(gpu, rs, sc, wave_paths=4096)
    assert np.array_equal(ca, cb)
    assert np.abs(a - b).max() <= 5e-6 * np.abs(a).max()


def test_masked_sky_scene(gpu, scenes):
    """Masked materials under the MIS estimator's environment rays."""
    sc = scenes.scene_c2(64, 36, 32, tri_scale=0.02, sky_size=(128, 64))
    sc = dataclasses.replace(sc, materials=[dataclasses.replace(m, alpha_mode=2, base_color=m.base_color[:3] + (0.0,)) if i % 3 == 0
                                            else m for i, m in enumerate(sc.materials)])
    rs = gpu.RenderScene(sc)
    for estimator in (0, 1):
        a, _ = _render(gpu, rs, sc, estimator=estimator)
        b, _ = _render(gpu, rs, sc, estimator=estimator, wave_paths=2048)
        assert np.array_equal(a, b)


@pytest.mark.parametrize("n", [1, 3, 129, 32768])
def test_traced_rays_do_not_depend_on_the_queue_length(gpu, scenes, n):
    """A few rays alone (eight lanes each) and among 33000 (one thread each): negative tnear, short and empty intervals,
    zero, axis-parallel and non-finite directions, masked materials."""
    sc = scenes.scene_textured(8, 8, 1)
    rng = np.random.default_rng(n)
    rs = gpu.RenderScene(sc)
    rays = np.zeros((33_000, 8), np.float32)
    rays[:, 0:3] = rng.uniform(-3, 3, (len(rays), 3)) + [0, 0, -4]
    rays[:, 4:7] = rng.normal(size=(len(rays), 3))
    rays[:, 7] = rng.choice([3e38, 2.0, 0.5], len(rays))
    rays[:, 3] = rng.choice([0.0, 0.0, 1.0, -2.0], len(rays))
    rays[rng.random(len(rays)) < 0.1, 4] = 0.0
    rays[rng.random(len(rays)) < 0.05, 5:7] = 0.0
    rays[::97, 4:7] = 0.0
    rays[1::211, 5] = np.nan
    rays[2::211, 6] = np.inf
    whole, alone = rs.trace(rays), rs.trace(rays[:n])
    assert (whole["inst"] != 0xFFFFFFFF).sum() > 5000
    assert np.array_equal(whole[:n].view(np.uint32), alone.view(np.uint32))
