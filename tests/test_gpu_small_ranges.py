"""The SAH build gives ranges of up to 8 triangles eight lanes each, of up to 32
a warp, and longer ones blocks of 128, 256 (from 257) and 1024 threads (from
2048), and makes nodes of pairs with their parents: hits of meshes at those
sizes are the oracle's, bit for bit."""
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


SHORT = [2, 3, 4, 7, 8, 9, 10, 16, 31, 32, 33, 34, 63, 65, 257]
LONG = [256, 258, 2047, 2048, 2049, 6007]


@pytest.mark.parametrize("sizes", [SHORT, LONG], ids=["short", "long"])
@pytest.mark.parametrize("kind", ["random", "equal", "line", "huge"])
def test_mesh_sizes_at_the_edges_of_the_classes(gpu, oracle, scenes, kind, sizes):
    rng = np.random.default_rng(31)
    base = scenes.scene_mixed(8, 8, 1)
    meshes, insts = [], []
    for k, nt in enumerate(sizes):
        v = rng.normal(size=(nt, 3, 3)).astype(np.float32) * np.float32(0.3)
        if kind == "equal":   # every split costs the same
            v[:] = v[:1]
        elif kind == "line":  # split off one end at a time: sizes of the triangles double
            v = v[:1] * np.float32(1.2) ** np.arange(nt, dtype=np.float32)[:, None, None] % 50
        elif kind == "huge":  # areas overflow: no best axis
            v[0] *= np.float32(1e19)
        v += rng.uniform(-3, 3, 3).astype(np.float32)
        meshes.append(scenes.Mesh(positions=v.reshape(-1, 3), normals=None,
                                  faces=np.arange(3 * nt, dtype=np.uint32).reshape(nt, 3),
                                  material=k % len(base.materials), name=f"m{k}"))
        t = np.eye(4, dtype=np.float32)
        t[2, 3] = -8
        insts.append(scenes.Instance(t, k))
    sc = dataclasses.replace(base, meshes=meshes, instances=insts)
    o = rng.uniform([-6, -6, -14], [6, 6, -2], (40_000, 3))
    d = rng.normal(size=o.shape)
    rays = np.zeros((len(o), 8), np.float32)
    rays[:, 0:3], rays[:, 4:7], rays[:, 7] = o, d / np.linalg.norm(d, axis=1, keepdims=True), 3.4e38
    a, b = gpu.RenderScene(sc).trace(rays), oracle.OracleScene(sc).trace(rays)
    assert (b["inst"] != 0xFFFFFFFF).any()
    for name in ("inst", "geom", "prim", "material", "t", "u", "v"):
        assert np.array_equal(a[name].view(np.uint32), b[name].view(np.uint32)), name


@pytest.mark.parametrize("sizes", [SHORT, LONG], ids=["short", "long"])
@pytest.mark.parametrize("octaves", [0, 12, 40])
def test_lines_of_growing_triangles(gpu, oracle, scenes, octaves, sizes):
    """Triangles along a line, each larger and farther out than the one before (by a factor of 2^(octaves / number), all
    of them finite): splits take one end off at a time, so a range goes through every class of sizes."""
    rng = np.random.default_rng(octaves)
    base = scenes.scene_mixed(8, 8, 1)
    meshes, insts = [], []
    for k, nt in enumerate(sizes):
        one = rng.normal(size=(1, 3, 3)) + rng.normal(size=3) * 3
        grow = 2.0 ** (octaves * (np.arange(nt) / nt - 0.5))
        v = (one * grow[:, None, None] * 0.1).astype(np.float32) + rng.uniform(-3, 3, 3).astype(np.float32)
        assert np.isfinite(v).all()
        meshes.append(scenes.Mesh(positions=v.reshape(-1, 3), normals=None,
                                  faces=np.arange(3 * nt, dtype=np.uint32).reshape(nt, 3),
                                  material=k % len(base.materials), name=f"m{k}"))
        t = np.eye(4, dtype=np.float32)
        t[2, 3] = -8
        insts.append(scenes.Instance(t, k))
    sc = dataclasses.replace(base, meshes=meshes, instances=insts)
    # rays past the triangles' centres, near and far, and anywhere
    centres = np.concatenate([m.positions.reshape(-1, 3, 3).mean(axis=1) + [0, 0, -8] for m in meshes])
    n = 40_000
    at = centres[rng.integers(0, len(centres), n)] * (1 + 0.05 * rng.normal(size=(n, 1)))
    o = rng.uniform([-6, -6, -14], [6, 6, -2], (n, 3))
    d = np.where(rng.random((n, 1)) < 0.7, at - o, rng.normal(size=o.shape))
    rays = np.zeros((n, 8), np.float32)
    rays[:, 0:3], rays[:, 4:7], rays[:, 7] = o, d / np.linalg.norm(d, axis=1, keepdims=True), 3.4e38
    a, b = gpu.RenderScene(sc).trace(rays), oracle.OracleScene(sc).trace(rays)
    assert (b["inst"] != 0xFFFFFFFF).sum() > 1000
    for name in ("inst", "geom", "prim", "material", "t", "u", "v"):
        assert np.array_equal(a[name].view(np.uint32), b[name].view(np.uint32)), name
