"""Renders of one scene in flight at the same time, each with its own counter
and samples: on two streams without a wait between, a larger frame enqueued
behind a smaller one, and beside a capture on another stream. Every image is
the one its render gives alone, bit for bit."""
import pytest

pytestmark = pytest.mark.gpu


class Frame:
    def __init__(self, built, scene, camera, w, h, spp, aux=False):
        import torch
        self.scene, self.camera = scene, camera
        self.st = built.Scene.settings(w, h, spp, 10, seed=w + spp)
        self.out = torch.full((h, w, 3), float("nan"), device="cuda")
        self.aux = torch.full((h, w, 7), float("nan"), device="cuda") if aux else None
        torch.cuda.synchronize()

    def enqueue(self, stream):
        self.scene.render_device(self.camera, self.st, self.out.data_ptr(),
                                 self.aux.data_ptr() if self.aux is not None else 0, 0, stream.cuda_stream)

    def images(self):
        return [t.view_as(t).cpu().numpy().tobytes() for t in (self.out, self.aux) if t is not None]


SIZES = [(640, 360, 1), (400, 225, 16), (1024, 1024, 24, True), (640, 360, 8), (1500, 1000, 2, True), (33, 17, 5)]


@pytest.mark.parametrize("kind,param", [(11, 4), (10, 40), (12, 200)])
def test_frames_in_flight_on_two_streams(built, kind, param):
    import torch
    g = built.Generated(kind, seed=3, param=param)
    want = []
    for size in SIZES:
        f = Frame(built, built.Scene(g), g.camera, *size)
        f.enqueue(torch.cuda.current_stream())
        torch.cuda.synchronize()
        want.append(f.images())
    s = built.Scene(g)
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    for _ in range(3):
        frames = [Frame(built, s, g.camera, *size) for size in SIZES]
        for k, f in enumerate(frames):
            f.enqueue(streams[k % 2])
        for st in streams:
            s.sync(st.cuda_stream)
        for f, w in zip(frames, want):
            assert f.images() == w


def test_render_beside_a_capture(built):
    import torch
    g = built.Generated(11, seed=3, param=3)
    s = built.Scene(g)
    alone = Frame(built, s, g.camera, 1024, 1024, 24)
    alone.enqueue(torch.cuda.current_stream())
    torch.cuda.synchronize()
    s2, other = built.Scene(g), torch.cuda.Stream()
    beside, captured = Frame(built, s2, g.camera, 1024, 1024, 24, True), Frame(built, s, g.camera, 320, 180, 4)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        captured.enqueue(torch.cuda.current_stream())
        beside.enqueue(other)
    graph.replay()
    torch.cuda.synchronize()
    assert beside.images()[0] == alone.images()[0]
    assert torch.isfinite(captured.out).all() and torch.isfinite(beside.aux).all()
