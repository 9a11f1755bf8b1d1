"""Frames and gradients captured into CUDA graphs, in every capture mode, while
other calls on the same handle go on: a captured call neither needs memory that
a capture may not allocate, nor shares streams or buffers with calls outside
it.  Films of lit scenes agree up to the order of the FP32 additions to a path's
radiance (5e-6), gradients up to the order of their sums (1e-4, as in
test_gpu_adjoint_waves.py)."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu
MODES = {"global": 0, "thread_local": 1, "relaxed": 2}


@pytest.fixture(scope="module")
def torch(gpu):
    return pytest.importorskip("torch")


class Graph:
    """A graph captured from a stream, and its instances (driver API)."""

    def __init__(self, torch, mode):
        self.cu = C.CDLL("libcuda.so.1")
        self.stream = torch.cuda.Stream()
        self.s = C.c_void_p(self.stream.cuda_stream)
        self.graph, self.execs = C.c_void_p(), []
        self.mode, self.capturing = MODES[mode], False

    def _ok(self, r):
        assert r == 0, f"CUDA driver error {r}"

    def __enter__(self):
        return self

    def __exit__(self, *error):
        if self.capturing:
            self.cu.cuStreamEndCapture(self.s, C.byref(self.graph))
            self.capturing = False
        self.destroy()

    def begin(self):
        self._ok(self.cu.cuStreamBeginCapture_v2(self.s, self.mode))
        self.capturing = True

    def end(self):
        self.capturing = False
        self._ok(self.cu.cuStreamEndCapture(self.s, C.byref(self.graph)))

    def instantiate(self):
        e = C.c_void_p()
        self._ok(self.cu.cuGraphInstantiateWithFlags(C.byref(e), self.graph, C.c_uint64(0)))
        self.execs.append(e)
        return e

    def launch(self, e):
        self._ok(self.cu.cuGraphLaunch(e, self.s))

    def destroy(self):
        for e in self.execs:
            self._ok(self.cu.cuGraphExecDestroy(e))
        if self.graph:
            self._ok(self.cu.cuGraphDestroy(self.graph))
        self.execs, self.graph = [], C.c_void_p()


class Frame:
    """omv_render_device of a scene with point lights into a film of its own per call."""

    rtol = 5e-6

    def __init__(self, gpu, scenes, torch, w=96, h=64, spp=8):
        self.gpu, self.torch = gpu, torch
        self.sc = scenes.scene_c1(w, h, spp)
        self.rs = gpu.RenderScene(self.sc)
        self.size(w, h, spp)

    def size(self, w, h, spp):
        cam = self.gpu.PinholeCamera.from_spec(self.sc.camera)
        cam.width, cam.height = w, h
        cam.adjust_to_resolution()
        cam.set_y_fov(45.0)
        self.cam = cam.to_c()
        self.prm = self.gpu.RendererParameters.for_scene(self.sc, samplesPerPixel=spp, seed=5).to_c()

    def buffers(self):
        return (self.torch.zeros((self.cam.height, self.cam.width, 3), dtype=self.torch.float64, device="cuda"),
                self.torch.zeros((self.cam.height, self.cam.width), dtype=self.torch.int32, device="cuda"))

    def call(self, stream, out):
        self.gpu.check(self.gpu.lib().omv_render_device(self.rs.handle, C.byref(self.cam), C.byref(self.prm),
                                                        C.c_void_p(out[0].data_ptr()), None, C.c_void_p(out[1].data_ptr()),
                                                        C.c_void_p(stream.cuda_stream), None))

    def check(self, out, want, times):
        assert int(out[1].min()) == int(out[1].max()) == times * self.prm.samples_per_pixel
        assert float((out[0] - times * want[0]).abs().max()) <= self.rtol * times * float(want[0].abs().max())


class Gradient:
    """omv_adjoint of a scene with point lights."""

    rtol = 1e-4

    def __init__(self, gpu, scenes, torch, side=48, spp=32):
        self.gpu, self.torch = gpu, torch
        self.sc = scenes.scene_materials(side, side, 1, tris=4_000, n_materials=4, bounces=4, seed=3)
        self.rs = gpu.RenderScene(self.sc)
        self.cam = gpu.PinholeCamera.from_spec(self.sc.camera).to_c()
        self.prm = gpu.RendererParameters.for_scene(self.sc, samplesPerPixel=spp, seed=11).to_c()
        self.adj = torch.rand((side, side, 3), device="cuda", generator=torch.Generator(device="cuda").manual_seed(5)) - 0.3

    def buffers(self):
        return (self.torch.zeros((len(self.sc.materials), 11), device="cuda"),)

    def call(self, stream, out):
        self.gpu.check(self.gpu.lib().omv_adjoint(self.rs.handle, C.byref(self.cam), C.byref(self.prm),
                                                  C.c_void_p(self.adj.data_ptr()), C.c_void_p(out[0].data_ptr()),
                                                  C.c_void_p(stream.cuda_stream)))

    def check(self, out, want, times):
        scale = float(want[0].abs().max())
        assert scale > 0
        assert float((out[0] - times * want[0]).abs().max()) <= self.rtol * times * scale


def _want(torch, work):
    out = work.buffers()
    work.call(torch.cuda.current_stream(), out)
    torch.cuda.synchronize()
    return out


@pytest.mark.parametrize("work", [Frame, Gradient])
def test_direct_calls_while_a_stream_is_captured(gpu, scenes, torch, work):
    """Another stream's calls before the capture ends run at once and leave it alone."""
    w = work(gpu, scenes, torch)
    want, direct, inside = _want(torch, w), w.buffers(), w.buffers()
    other = torch.cuda.Stream()
    torch.cuda.synchronize()
    with Graph(torch, "relaxed") as g:
        g.begin()
        w.call(g.stream, inside)
        w.call(other, direct)
        other.synchronize()
        w.call(g.stream, inside)  # and on in the capture
        w.call(other, direct)
        other.synchronize()
        g.end()
        w.check(direct, want, 2)
        g.launch(g.instantiate())
        torch.cuda.synchronize()
        w.check(inside, want, 2)


@pytest.mark.parametrize("work", [Frame, Gradient])
def test_two_streams_captured_at_once(gpu, scenes, torch, work):
    w = work(gpu, scenes, torch)
    want, a, b = _want(torch, w), w.buffers(), w.buffers()
    torch.cuda.synchronize()
    with Graph(torch, "relaxed") as ga, Graph(torch, "relaxed") as gb:
        ga.begin()
        w.call(ga.stream, a)
        gb.begin()
        w.call(gb.stream, b)
        w.call(ga.stream, a)
        ga.end()
        w.call(gb.stream, b)
        gb.end()
        for g in (ga, gb):
            g.launch(g.instantiate())
            torch.cuda.synchronize()
        w.check(a, want, 2)
        w.check(b, want, 2)


# 2^22 paths each, so that one scratch serves all three: 8192 tiles of 512 pixels, 8192 and 131072
MANY_TILES = [(2048, 2048, 1), (65536, 64, 1), (4194304, 1, 1)]


@pytest.mark.parametrize("mode", MODES)
def test_captured_frame_with_more_tiles_than_any_before(gpu, scenes, torch, mode):
    w = Frame(gpu, scenes, torch, *MANY_TILES[0])
    _want(torch, w)
    w.size(*MANY_TILES[2])
    out = w.buffers()
    torch.cuda.synchronize()
    with Graph(torch, mode) as g:
        g.begin()
        w.call(g.stream, out)
        g.end()
        e0, e1 = g.instantiate(), g.instantiate()
        for e in (e0, e1):
            g.launch(e)
        torch.cuda.synchronize()
        w.check(out, _want(torch, w), 2)


def test_direct_frames_of_more_tiles_between_replays(gpu, scenes, torch):
    """A captured frame's tile lists are made by its replay: direct frames with more tiles, before the capture ends and
    between replays, change nothing."""
    w = Frame(gpu, scenes, torch, *MANY_TILES[0])
    want, out = _want(torch, w), w.buffers()
    other = torch.cuda.Stream()
    w.size(*MANY_TILES[2])
    more = w.buffers()
    w.size(*MANY_TILES[0])
    torch.cuda.synchronize()
    with Graph(torch, "relaxed") as g:
        g.begin()
        w.call(g.stream, out)
        w.size(*MANY_TILES[2])
        w.call(other, more)
        other.synchronize()
        g.end()
        e = g.instantiate()
        for _ in range(2):
            g.launch(e)
            w.call(g.stream, more)
        torch.cuda.synchronize()
        w.check(more, _want(torch, w), 3)
        w.size(*MANY_TILES[0])
        w.check(out, want, 2)


def test_captures_one_after_another_use_the_same_memory(gpu, scenes, torch):
    """64 graphs of frames with 36 MB of tile lists each leave less than three times that behind."""
    w = Frame(gpu, scenes, torch, *MANY_TILES[2])
    out = w.buffers()
    _want(torch, w)
    torch.cuda.synchronize()
    free0 = torch.cuda.mem_get_info()[0]
    for _ in range(64):
        with Graph(torch, "thread_local") as g:
            g.begin()
            w.call(g.stream, out)
            g.end()
            g.launch(g.instantiate())
            torch.cuda.synchronize()
    assert free0 - torch.cuda.mem_get_info()[0] < 3 * 36 * 2**20
    w.check(out, _want(torch, w), 64)


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("work", [Frame, Gradient])
def test_two_instances_of_a_graph(gpu, scenes, torch, work, mode):
    """A captured call has no memory nodes: its graph is instantiated twice, in every capture mode."""
    w = work(gpu, scenes, torch)
    want, out, direct = _want(torch, w), w.buffers(), w.buffers()
    torch.cuda.synchronize()
    with Graph(torch, mode) as g:
        g.begin()
        w.call(g.stream, out)
        g.end()
        e0, e1 = g.instantiate(), g.instantiate()
        for e in (e0, e1, e0):
            g.launch(e)
        torch.cuda.synchronize()
        w.call(g.stream, direct)
        g.launch(e1)
        torch.cuda.synchronize()
        w.check(out, want, 4)
        w.check(direct, want, 1)


def test_instances_and_direct_gradients_on_their_own_streams(gpu, scenes, torch):
    """A graph of three gradients, two of them on branches side by side, as two instances on two streams with direct
    calls on a third, none waiting for another: each has its records to itself while it runs."""
    w = Gradient(gpu, scenes, torch, side=64, spp=64)
    want, out, direct = _want(torch, w), w.buffers(), w.buffers()
    streams = [torch.cuda.Stream() for _ in range(3)]
    branch, fork, join = torch.cuda.Stream(), torch.cuda.Event(), torch.cuda.Event()
    torch.cuda.synchronize()
    with Graph(torch, "relaxed") as g:
        g.begin()
        w.call(g.stream, out)
        fork.record(g.stream)
        branch.wait_event(fork)
        w.call(branch, out)
        join.record(branch)
        w.call(g.stream, out)
        g.stream.wait_event(join)
        g.end()
        execs = [g.instantiate(), g.instantiate()]
        for _ in range(20):
            for e, st in zip(execs, streams):
                g._ok(g.cu.cuGraphLaunch(e, C.c_void_p(st.cuda_stream)))
            w.call(streams[2], direct)
        torch.cuda.synchronize()
        w.check(out, want, 120)
        w.check(direct, want, 20)


def test_gradients_of_two_handles_in_one_capture(gpu, scenes, torch):
    """Two handles on branches side by side, one graph after another: blocks of graphs that are gone serve the next capture
    and the direct calls, of either handle."""
    a, b = Gradient(gpu, scenes, torch, side=96, spp=32), Gradient(gpu, scenes, torch, side=40, spp=20)
    wa, wb, oa, ob = _want(torch, a), _want(torch, b), a.buffers(), b.buffers()
    branch, fork, join = torch.cuda.Stream(), torch.cuda.Event(), torch.cuda.Event()
    torch.cuda.synchronize()
    for _ in range(6):
        with Graph(torch, "thread_local") as g:
            g.begin()
            fork.record(g.stream)
            branch.wait_event(fork)
            a.call(g.stream, oa)
            b.call(branch, ob)
            b.call(branch, ob)
            join.record(branch)
            a.call(g.stream, oa)
            g.stream.wait_event(join)
            g.end()
            e0, e1 = g.instantiate(), g.instantiate()
            for _ in range(3):
                g.launch(e0)
                g._ok(g.cu.cuGraphLaunch(e1, C.c_void_p(branch.cuda_stream)))
            torch.cuda.synchronize()
        a.call(g.stream, oa)
        b.call(branch, ob)
    torch.cuda.synchronize()
    a.check(oa, wa, 6 * 13)
    b.check(ob, wb, 6 * 13)


def test_gradients_of_one_capture_share_their_records(gpu, scenes, torch):
    """Graphs of 16 gradients of 1.2 GB of records each, one graph after another, leave less than 3 GiB behind."""
    w = Gradient(gpu, scenes, torch, side=128, spp=64)
    want, out = _want(torch, w), w.buffers()
    torch.cuda.synchronize()
    free0 = torch.cuda.mem_get_info()[0]
    for _ in range(8):
        with Graph(torch, "thread_local") as g:
            g.begin()
            for _ in range(16):
                w.call(g.stream, out)
            g.end()
            g.launch(g.instantiate())
            torch.cuda.synchronize()
    assert free0 - torch.cuda.mem_get_info()[0] < 3 * 2**30
    w.check(out, want, 128)


def test_clone_and_child_graph_keep_the_records(gpu, scenes, torch):
    """A clone of a captured gradient and a graph that holds it as a child outlive the captured graph, with its records:
    direct calls and another capture in between have their own."""
    w = Gradient(gpu, scenes, torch)
    want, out, other = _want(torch, w), w.buffers(), w.buffers()
    torch.cuda.synchronize()
    with Graph(torch, "relaxed") as clone, Graph(torch, "relaxed") as parent:
        with Graph(torch, "relaxed") as g:
            g.begin()
            w.call(g.stream, out)
            g.end()
            g._ok(g.cu.cuGraphClone(C.byref(clone.graph), g.graph))
            g._ok(g.cu.cuGraphCreate(C.byref(parent.graph), 0))
            node = C.c_void_p()
            g._ok(g.cu.cuGraphAddChildGraphNode(C.byref(node), parent.graph, None, C.c_size_t(0), g.graph))
        ec, ep = clone.instantiate(), parent.instantiate()
        with Graph(torch, "relaxed") as later:
            later.begin()
            w.call(later.stream, other)
            later.end()
            el = later.instantiate()
            for _ in range(5):
                clone.launch(ec)
                parent.launch(ep)
                later.launch(el)
                w.call(torch.cuda.current_stream(), other)
            torch.cuda.synchronize()
        w.check(out, want, 10)
        w.check(other, want, 10)
