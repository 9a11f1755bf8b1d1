"""Device image development (post.cu through the C ABI) against the
reference's outputs (tests/golden/post.npz) and the oracle's restatement:
the median and the 8-bit conversion are bit-exact; gamma correction agrees to
2e-6 relative, the error bound of the device powf against the host's."""
import importlib

import numpy as np
import pytest
from conftest import golden

pytestmark = pytest.mark.gpu

TONEMAP_RTOL = 2e-6


@pytest.fixture(scope="module")
def post(gpu):
    torch = pytest.importorskip("torch")
    return torch, importlib.import_module("openmaterial-validation_gb300.post")


def _dev(torch, a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _host(torch, t):
    torch.cuda.synchronize()
    return t.cpu().numpy()


@pytest.mark.parametrize("name,gamma", [("tonemap_0.5", 0.5), ("tonemap_0.4545", 0.4545)])
def test_gamma_correction_matches_reference(post, name, gamma):
    torch, P = post
    g = golden("post")
    y = _host(torch, P.gammaCorrection(_dev(torch, g["image"]), 1.0, gamma))
    ref = g[name]
    assert np.all(y[..., 3] == 1.0)
    assert np.all(np.abs(y - ref) <= TONEMAP_RTOL * np.abs(ref)), np.max(np.abs(y - ref) / np.maximum(ref, 1e-30))
    # clamped and black pixels are exact
    sat = (ref == 1.0) | (ref == 0.0)
    assert np.array_equal(y[sat], ref[sat])


def test_median_matches_reference(post):
    torch, P = post
    g = golden("post")
    y = _host(torch, P.SimpleDenoiserMedian(_dev(torch, g["tonemap_0.5"]), 1))
    assert np.array_equal(y, g["median"])


@pytest.mark.parametrize("half", [1, 2, 3])
@pytest.mark.parametrize("shape", [(7, 5), (67, 45), (300, 171)])
def test_median_matches_oracle_on_ragged_sizes(post, oracle, half, shape):
    torch, P = post
    rng = np.random.default_rng(half * 1000 + shape[0])
    img = rng.uniform(0, 1, shape + (4,)).astype(np.float32)
    img[..., :3] = np.round(img[..., :3] * 16) / 16  # many ties
    y = _host(torch, P.SimpleDenoiserMedian(_dev(torch, img), half))
    assert np.array_equal(y, oracle.median(img, half))


@pytest.mark.parametrize("half", [1, 2, 3])
@pytest.mark.parametrize("shape", [(1, 1), (2, 9), (3, 3), (5, 129), (9, 128), (130, 7)])
def test_median_edges_and_infinities(post, oracle, half, shape):
    """Row groups and column blocks cut short, windows that do not fit, infinite pixels: exact."""
    torch, P = post
    rng = np.random.default_rng(17 * half + shape[1])
    img = rng.lognormal(0.0, 2.0, shape + (4,)).astype(np.float32)
    img[rng.random(shape) < 0.05] = np.inf
    y = _host(torch, P.SimpleDenoiserMedian(_dev(torch, img), half))
    assert np.array_equal(y, oracle.median(img, half))


def test_median3_of_windows_with_nan(post):
    """A NaN in the window: the result of the 19-exchange network with IEEE minimum and maximum numbers."""
    torch, P = post
    rng = np.random.default_rng(3)
    img = rng.uniform(0, 1, (23, 41, 4)).astype(np.float32)
    img[rng.random((23, 41)) < 0.05] = np.nan
    H, W = img.shape[:2]
    p = [img[dy:H - 2 + dy, dx:W - 2 + dx, :3].copy() for dy in range(3) for dx in range(3)]
    for a, b in [(1, 2), (4, 5), (7, 8), (0, 1), (3, 4), (6, 7), (1, 2), (4, 5), (7, 8), (0, 3), (5, 8), (4, 7), (3, 6),
                 (1, 4), (2, 5), (4, 7), (4, 2), (6, 4), (4, 2)]:
        p[a], p[b] = np.fmin(p[a], p[b]), np.fmax(p[a], p[b])
    y = _host(torch, P.SimpleDenoiserMedian(_dev(torch, img), 1))
    assert np.array_equal(y[1:-1, 1:-1, :3], p[4], equal_nan=True)


@pytest.mark.parametrize("shape", [(1, 1), (3, 257), (512, 2048)])
def test_develop_equals_the_fp64_expression(post, shape):
    """(float)(sum * (1.0 / count)) bit for bit: counts up to 2^31, sums of any size and sign, zeros, infinities, and
    sums whose quotient lies within an FP64 ulp or two of the middle between two floats."""
    torch, P = post
    rng = np.random.default_rng(shape[1])
    count = rng.choice([0, 1, 3, 64, 1000, 2**24 - 1, 2**24 + 1, 2**31 - 1], shape).astype(np.int32)
    count = np.where(rng.random(shape) < 0.5, rng.integers(1, 300, shape), count).astype(np.int32)
    c = np.maximum(count, 1).astype(np.float64)[..., None]
    s = rng.lognormal(0.0, 3.0, shape + (3,))
    f = rng.lognormal(0.0, 3.0, shape + (3,)).astype(np.float32)
    tie = (f.astype(np.float64) + np.nextafter(f, np.float32(np.inf)).astype(np.float64)) / 2 * c
    tie = tie * (1.0 + rng.integers(-3, 4, tie.shape) * 2.0**-52)
    s = np.where(rng.random(s.shape) < 0.3, tie, s)
    s = np.where(rng.random(s.shape) < 0.1, -s, s)
    special = np.array([0.0, -0.0, np.inf, 1e-310, 5e-324, 1e-44, 1e30, 1e37, 3e38, 1e300, 2.0**-70, 2.0**-71, 2.0**90, 2.0**91])
    s = np.where(rng.random(s.shape) < 0.1, rng.choice(special, s.shape), s)
    lin = _host(torch, P.develop(_dev(torch, s), _dev(torch, count), tonemapped=False, rgba8=False)["linear"])
    with np.errstate(over="ignore"):
        want = (s * np.where(count[..., None] < 1, 1.0, 1.0 / c)).astype(np.float32)
    assert np.array_equal(lin[..., :3].view(np.uint32), want.view(np.uint32))


def test_rgba8_matches_reference(post):
    torch, P = post
    g = golden("post")
    x = _dev(torch, g["tonemap_0.5"])
    assert np.array_equal(_host(torch, P.rgba8(x)), g["rgba8"])
    assert np.array_equal(_host(torch, P.rgba8(x, flip=True)), g["rgba8"][::-1])


def test_develop_matches_resolve_tonemap_and_conversion(post, oracle):
    torch, P = post
    rng = np.random.default_rng(5)
    H, W = 131, 77
    count = rng.integers(0, 40, (H, W)).astype(np.int32)
    s = (rng.lognormal(-1.0, 1.5, (H, W, 3)) * count[..., None]).astype(np.float64)
    out = P.develop(_dev(torch, s), _dev(torch, count), gamma=0.5)
    lin = _host(torch, out["linear"])
    c = count.astype(np.float64)[..., None]
    want = np.concatenate([(s * np.where(c < 0.5, 1.0, 1.0 / np.maximum(c, 1))).astype(np.float32),
                           np.ones((H, W, 1), np.float32)], axis=-1)
    assert np.array_equal(lin, want)
    ref = oracle.tonemap(lin, 0.5)
    tm = _host(torch, out["tonemapped"])
    assert np.all(np.abs(tm - ref) <= TONEMAP_RTOL * np.abs(ref))
    assert np.array_equal(_host(torch, out["rgba8"]), _host(torch, P.rgba8(out["tonemapped"], flip=True)))


def test_develop_of_a_render_equals_the_render_image(post, gpu, scenes):
    """omv_develop's linear image of a device film is omv_render's image."""
    torch, P = post
    sc = scenes.scene_c1(64, 48, 4)
    rs = gpu.RenderScene(sc)
    r = gpu.BDPTRenderer()
    r.set_parameters(gpu.RendererParameters.for_scene(sc, seed=3))
    r.set_scene(rs)
    img, s, _, cnt = r.render(gpu.PinholeCamera.from_spec(sc.camera), sums=True)
    out = P.develop(_dev(torch, s), _dev(torch, cnt.astype(np.int32)), linear=True, tonemapped=False, rgba8=False)
    assert np.array_equal(_host(torch, out["linear"]), img)


def test_full_hd_properties(post, oracle):
    """1920x1080: gamma 1 is the clamp alone, and the median equals the oracle's."""
    torch, P = post
    rng = np.random.default_rng(8)
    img = rng.lognormal(-1.0, 1.0, (1080, 1920, 4)).astype(np.float32)
    x = _dev(torch, img)
    y = _host(torch, P.gammaCorrection(x.clone(), 1.0, 1.0))
    want = np.clip(img, 0, 1)
    want[..., 3] = 1.0
    assert np.array_equal(y, want)
    t = oracle.tonemap(img, 0.5)
    m = _host(torch, P.SimpleDenoiserMedian(_dev(torch, t), 1))
    assert np.array_equal(m, oracle.median(t, 1))


def test_argument_errors(post, gpu):
    torch, P = post
    L = gpu.lib()
    x = torch.zeros((4, 4, 4), dtype=torch.float32, device="cuda")
    with pytest.raises(gpu.OmvError, match="half"):
        P.SimpleDenoiserMedian(x, 4)
    assert L.omv_denoise_median(x.data_ptr(), x.data_ptr(), 4, 4, 1, None) == 1
    assert L.omv_develop(None, None, 4, 4, 1.0, 0.5, None, None, None, 0, None) == 1
    assert L.omv_rgba8(x.data_ptr(), None, 4, 4, 0, None) == 1
    assert L.omv_tonemap(x.data_ptr(), 0, 1.0, 0.5, None) == 0
