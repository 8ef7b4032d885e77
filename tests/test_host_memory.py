"""What the library's host code does with device memory -- allocations that
fail, buffers that renders share, what is kept -- on the CPU, over a fake CUDA
runtime that logs every launch and whether its buffers are allocated."""
import ctypes as C

import pytest

from host_library import Fake, build_fake


@pytest.fixture(scope="module")
def fake_library(tmp_path_factory):
    return Fake(build_fake(str(tmp_path_factory.mktemp("fake"))))


@pytest.fixture
def fake(fake_library, monkeypatch):
    from photon_tracer_b200 import abi
    monkeypatch.setattr(abi, "_lib", fake_library.lib)
    fake_library.fail_after(-1)
    fake_library.log()
    yield fake_library
    fake_library.fail_after(-1)


SOME = C.c_void_p(64)  # a caller's device pointer; no fake kernel reads it


def denoise(fake, net, w, h):
    return fake.lib.pt_denoise_unet(net, w, h, SOME, SOME, SOME, SOME, None)


def grads(fake, net, b, h, w):
    return fake.lib.pt_unet_loss_grads(net, b, h, w, SOME, SOME, None, None, None)


@pytest.mark.parametrize("call,sizes", [(denoise, (200, 104)), (denoise, (33, 17)), (grads, (2, 24, 40))])
@pytest.mark.parametrize("tensor_cores", [1, 0])
def test_unet_after_a_failed_allocation(fake, call, sizes, tensor_cores):
    """A call that ran out of memory leaves nothing behind that a later call of the same size takes for its
    workspace: that call fails too while there is no memory, and otherwise allocates what is missing."""
    from photon_tracer_b200 import abi
    failures = 0
    for k in range(200):
        net = C.c_void_p()
        abi.check(fake.lib.pt_unet_create(1, C.byref(net)))
        fake.lib.pt_unet_set_tensor_cores(net, tensor_cores)
        fake.fail_after(k)
        first = call(fake, net, *sizes)
        second = call(fake, net, *sizes)
        fake.fail_after(-1)
        third = call(fake, net, *sizes)
        bad = [line for line in fake.log() if line.startswith("bad")]
        fake.lib.pt_unet_destroy(net)
        assert not bad, (k, bad[:3])
        assert third == abi.PT_OK
        if first == abi.PT_OK:
            break
        assert first == second == abi.PT_ERR_OUT_OF_MEMORY
        failures += 1
    assert failures > 10


class DeviceScene:
    """A generated scene whose renders go to the fake's log."""

    def __init__(self, kind, param):
        import photon_tracer_b200 as pt
        self.g = pt.Generated(kind, seed=1, param=param)
        self.s = pt.Scene(self.g)

    def render(self, w, h, spp, stream, aux=False, mode=1):
        st = self.s.settings(w, h, spp, 10, seed=1, mode=mode)
        self.s.render_device(self.g.camera, st, SOME.value, SOME.value if aux else 0, 0, stream)


def launches(lines, kind):
    """(stream, work counter, buffer or None) of the logged megakernel launches of one form."""
    out = []
    for line in lines:
        w = line.split()
        if w[0] == kind:
            out.append((w[1], w[3], w[5] if len(w) > 5 else None))
    return out


ROOM, SPHERES = 11, 10  # large enough trees to stream at any sample count from two; small ones from four


@pytest.mark.parametrize("kind,param,spp,form", [(ROOM, 4, 4, "samples"), (SPHERES, 20, 1, "megakernel")])
def test_renders_on_two_streams_share_nothing(fake, kind, param, spp, form):
    """Frames of one scene enqueued on two streams, neither waited for: each has its own counter and samples until
    its own launches are done."""
    d = DeviceScene(kind, param)
    fake.log()
    a, b = 0x7000, 0x8000
    d.render(400, 300, spp, a)
    d.render(320, 200, spp, b)
    lines = fake.log()
    on_a, on_b = launches(lines, form)
    assert (int(on_a[0], 16), int(on_b[0], 16)) == (a, b)
    assert on_a[1] != on_b[1] and (form == "megakernel" or on_a[2] != on_b[2])
    assert not any(line.startswith("bad") for line in lines)


def test_a_device_render_does_not_wait(fake):
    """Neither the first frame nor larger ones after it, nor guides, free memory or wait for the device; a frame that
    an earlier one's memory is large enough for allocates none."""
    d = DeviceScene(ROOM, 4)
    fake.log()
    new = []
    for w, h, spp, aux in ((64, 48, 4, False), (640, 360, 8, False), (1024, 1024, 24, True), (33, 17, 2, False),
                           (1024, 1024, 24, True), (640, 360, 8, True)):
        d.render(w, h, spp, 0x7000, aux)
        lines = fake.log()
        assert not [x for x in lines if x.split()[0] in ("free", "wait", "stream", "bad")], lines
        new.append(sum(x.startswith("malloc") for x in lines))
    assert new == [1, 1, 1, 0, 0, 0]


def test_scenes_hold_no_samples_between_renders(fake):
    """Scenes that render one after another do so in the same memory, whichever streams they use once the work is
    done, and the last of them frees it."""
    before = fake.live_bytes()
    scenes = [DeviceScene(ROOM, 3) for _ in range(4)]
    fake.log()
    for k, d in enumerate(scenes):
        if k == 3:
            fake.lib.fake_finish()
        d.render(640, 360, 8, 0x8000 if k == 3 else 0x7000)
    lines = fake.log()
    assert sum(x.startswith("malloc") for x in lines) == 1
    for d in scenes:
        assert fake.live_bytes() > before
        d.s.close()
    assert fake.live_bytes() == before


def test_memory_of_frames_in_flight_is_bounded(fake):
    """Large frames on many streams get memory of their own up to a bound; then a stream waits for another's, in
    stream order, and no frame goes without."""
    d = DeviceScene(ROOM, 3)
    before = fake.live_bytes()
    fake.log()
    streams = [0x7000 + 16 * k for k in range(10)]
    for stream in streams:
        d.render(1024, 1024, 22, stream)
    lines = fake.log()
    assert len(launches(lines, "samples")) >= 10 and not launches(lines, "megakernel")
    assert fake.live_bytes() - before <= 1280 << 20
    waits = [x.split()[2] for x in lines if x.startswith("stream waits")]
    assert waits and set(int(w, 16) for w in waits) <= set(streams[4:])
    assert len({buffer for _, _, buffer in launches(lines, "samples")}) == 10 - len(waits)


def test_captured_and_memoryless_renders_borrow_no_samples(fake):
    import numpy as np
    import photon_tracer_b200 as pt
    d = DeviceScene(ROOM, 4)
    fake.lib.fake_capture(0x7000)
    fake.log()
    d.render(400, 300, 4, 0x7000)
    fake.lib.fake_capture(None)
    lines = fake.log()
    assert len(launches(lines, "megakernel")) == 1 and not any(x.startswith("malloc") for x in lines)
    with fake.failing_above(1 << 20):
        d.render(400, 300, 4, 0x7000)
    with fake.failing_above(0):
        d.render(400, 300, 4, 0x7000)
    with fake.failing_above(3 * 4 * 400):  # a scanline's pixels, not its samples
        row = np.empty((400, 3), np.float32)
        pt.render_row_linear(d.s, d.g.camera, 3, 400, 300, 16, 10, row, 1)
    lines = fake.log()
    assert len(launches(lines, "megakernel")) == 3 and not launches(lines, "samples")
    assert not any(x.startswith("bad") for x in lines)


BATCH_SAMPLES = 4 * 256 * 256 * 4 * 12  # bytes of make_batch()'s samples at least
ONE_LAUNCH, PER_SCENE_MEGA, PER_SCENE_WAVE, AUTO = 1, 2, 3, 0


def make_batch(strategy, side=256, spp=4, max_bounces=10):
    """Four rooms; at the default size the single launch streams."""
    import photon_tracer_b200 as pt
    items = []
    for k in range(4):
        g = pt.Generated(ROOM, seed=k + 1, param=3)
        items.append((g, g.camera, side, side, spp, k))
    return pt.Batch(items, strategy, max_bounces=max_bounces)


def one_launch_lines(fake, batch):
    fake.log()
    batch.render()
    return [x for x in fake.log() if x.startswith(("batch", "bad"))]


@pytest.mark.parametrize("strategy", [PER_SCENE_MEGA, PER_SCENE_WAVE])
def test_per_scene_batches_hold_no_samples(fake, strategy):
    before = fake.live_bytes()
    b = make_batch(strategy)
    held = b.info().device_bytes
    assert fake.live_bytes() - before < BATCH_SAMPLES and held < BATCH_SAMPLES
    b.close()
    assert fake.live_bytes() == before


def test_batch_without_memory_for_its_samples(fake):
    """Whatever allocation fails, a batch either is refused and leaves nothing, or renders in lock step and holds no
    samples; one that is made streams when all succeed."""
    before, forms = fake.live_bytes(), []
    for k in range(10):
        fake.fail_after(k)
        try:
            b = make_batch(ONE_LAUNCH)
        except Exception:
            fake.fail_after(-1)
            assert fake.live_bytes() == before
            continue
        fake.fail_after(-1)
        forms += one_launch_lines(fake, b)
        if forms[-1] != "batch stream":
            assert fake.live_bytes() - before < BATCH_SAMPLES
        b.close()
        assert fake.live_bytes() == before
        if forms[-1] == "batch stream":
            break
    assert forms == ["batch 128", "batch stream"]


def test_batch_scenes_come_before_its_samples(fake):
    """A batch that needs its per-scene scenes is accepted in the memory that they and its arena take."""
    before = fake.live_bytes()
    small = make_batch(AUTO, max_bounces=0)  # nothing to stream
    need = fake.live_bytes() - before
    small.close()
    with fake.budget(before + need + BATCH_SAMPLES - 4096):
        b = make_batch(AUTO)
        assert one_launch_lines(fake, b)[0].split()[1] != "stream"
    b.close()


def test_a_tuned_batch_keeps_only_what_its_choice_needs(fake):
    before = fake.live_bytes()
    b = make_batch(AUTO, side=260)
    assert fake.live_bytes() - before > BATCH_SAMPLES
    with fake.falling_times():
        b.render()
    info = b.info()
    assert info.strategy == PER_SCENE_WAVE and info.device_bytes < BATCH_SAMPLES
    b.close()
    assert fake.live_bytes() == before


def test_autotuner_times_the_streaming_launch_once(fake):
    """The streaming form has one block shape: it is captured and timed as one candidate, whose time stands for all
    three, and its choice is not taken for a batch of the same totals that renders in lock step."""
    b = make_batch(AUTO, side=264)
    fake.log()
    b.render()
    assert fake.log().count("captured") == 1
    info = b.info()
    assert info.tuned and info.strategy == ONE_LAUNCH and info.threads == 128
    assert info.tune_ms[0] == info.tune_ms[1] == info.tune_ms[2] > 0
    b.close()
    b = make_batch(AUTO, side=264, max_bounces=0)
    fake.log()
    b.render()
    assert fake.log().count("captured") == 3 and all(ms > 0 for ms in b.info().tune_ms[:7])
    b.close()


def test_each_scene_keeps_its_own_launch_shapes(fake):
    """What a launch works out once belongs to its scene and form, as scenes may be on other devices and rendered by
    other threads."""
    a, b = DeviceScene(ROOM, 3), DeviceScene(ROOM, 3)
    fake.log()
    for d, aux, new in ((a, False, 1), (a, False, 0), (a, True, 1), (b, False, 1), (a, True, 0), (b, False, 0)):
        d.render(320, 200, 4, 0x7000, aux)
        assert fake.log().count("blocks worked out") == new


def test_a_scene_that_fits_only_without_its_second_nodes_is_accepted(fake):
    """The streaming walks' copy of the nodes is left out where it does not fit: the scene and the batch are made, and
    render in lock step. Scenes that cannot stream (leaves past a stack word, no tree) hold no copy."""
    import photon_tracer_b200 as pt
    before = fake.live_bytes()
    d = DeviceScene(ROOM, 4)
    full, nodes = d.s.info().device_bytes, 128 * d.s.info().n_nodes
    assert fake.live_bytes() - before == full
    d.s.close()
    with fake.budget(before + full - 4096):
        d = DeviceScene(ROOM, 4)
        assert d.s.info().device_bytes == full - (nodes + 255) // 256 * 256
    fake.log()
    d.render(320, 200, 16, 0x7000)
    assert not launches(fake.log(), "samples")
    d.s.close()
    b = make_batch(ONE_LAUNCH, max_bounces=0)
    arena = fake.live_bytes() - before
    b.close()
    with fake.budget(before + arena - 4096):
        b = make_batch(ONE_LAUNCH)
    assert one_launch_lines(fake, b) == ["batch 128"]
    b.close()
    assert pt.Scene(pt.Generated(0, seed=1)).info().n_nodes == 0 and "build_qnodes" not in fake.log()


def test_inference_allocates_nothing_for_the_backward(fake):
    """The buffers that only the tensor-core backward uses come with the first gradients of a size: two bf16 buffers'
    worth of the largest activation, one of which the workspace has, and 16 bytes per pixel."""
    from photon_tracer_b200 import abi
    net = C.c_void_p()
    abi.check(fake.lib.pt_unet_create(1, C.byref(net)))
    pixels = 2 * 64 * 40
    abi.check(fake.lib.pt_unet_forward(net, 2, 64, 40, SOME, SOME, None))
    inference = fake.live_bytes()
    assert grads(fake, net, 2, 64, 40) == abi.PT_OK
    assert fake.live_bytes() - inference == pixels * 32 * 2 + pixels * 16
    fake.lib.pt_unet_destroy(net)


# Scenes by (generator, parameter): 24 and 488 spheres and the reference's field under the sky, its room, rooms with
# 1,280 and 81,920 triangles, 300 instances under the sky.
SPHERES_24, SPHERES_488, FIELD, REF_ROOM, ROOM_1K, ROOM_80K, INSTANCES = (
    (10, 20), (10, 0), (1, 0), (3, 0), (11, 3), (11, 6), (12, 300))


@pytest.mark.parametrize("scene,streams,not_streams", [
    # (width, height, samples, bounces, guides)
    (SPHERES_24, [(640, 360, 8, 10, 0), (128, 72, 4, 10, 1)], [(1280, 720, 8, 10, 0), (640, 360, 3, 10, 0),
                                                             (640, 360, 8, 2, 0), (640, 360, 4, 3, 0)]),
    (SPHERES_488, [(400, 225, 16, 10, 0), (1920, 1080, 8, 10, 0), (1280, 720, 8, 10, 1)],
     [(1920, 1080, 8, 10, 1), (1280, 720, 3, 10, 0), (640, 360, 8, 1, 0)]),
    (FIELD, [(640, 360, 4, 10, 1)], [(1920, 1080, 8, 10, 0), (1280, 720, 4, 10, 0)]),
    (REF_ROOM, [(1920, 1080, 4, 3, 0), (640, 360, 4, 10, 1)], [(640, 360, 8, 1, 0), (640, 360, 8, 2, 1),
                                                            (1920, 1080, 4, 2, 0), (640, 360, 3, 10, 0),
                                                            (400, 225, 4, 2, 0)]),
    (ROOM_1K, [(640, 360, 2, 10, 0), (256, 256, 16, 1, 0), (1920, 1080, 1, 10, 0), (640, 360, 8, 1, 0)],
     [(640, 360, 8, 2, 0), (640, 360, 2, 1, 0), (1920, 1080, 4, 1, 0), (640, 360, 1, 10, 0)]),
    (ROOM_80K, [(1024, 1024, 64, 10, 0), (640, 360, 8, 1, 0), (640, 360, 8, 2, 0)],
     [(1920, 1080, 4, 1, 1), (1920, 1080, 4, 2, 0), (320, 180, 3, 2, 0)]),
    (INSTANCES, [(960, 540, 16, 10, 0), (640, 360, 2, 10, 0)], [(1920, 1080, 4, 1, 0)]),
])
def test_which_frames_stream(fake, scene, streams, not_streams):
    """Frames take the form that was measured faster for frames like them."""
    d = DeviceScene(*scene)
    for sizes, form in ((streams, "samples"), (not_streams, "megakernel")):
        for w, h, spp, depth, aux in sizes:
            st = d.s.settings(w, h, spp, depth, seed=1)
            fake.log()
            d.s.render_device(d.g.camera, st, SOME.value, SOME.value if aux else 0, 0, 0x7000)
            assert launches(fake.log(), form), (w, h, spp, depth, aux, form)


def test_lock_step_renders_borrow_nothing_on_their_usual_streams(fake):
    """A stream's lock-step renders count in that stream's own word, captured ones in another; with more streams than
    words, or no memory to borrow, the render still runs."""
    d = DeviceScene(SPHERES, 20)
    fake.log()
    work, streams = [{}, {}], [0x7000 + 16 * k for k in range(40)]
    for seen in work:
        for stream in streams:
            d.render(100, 60, 1, stream)
            lines = fake.log()
            ((_, seen[stream], _),) = launches(lines, "megakernel")
            assert ("malloc 1048576" in lines) == (stream >= streams[31] and seen is work[0])
    assert work[0] == work[1] and len(set(work[0].values())) == 40
    fake.lib.fake_capture(0x7000)
    d.render(100, 60, 1, 0x7000)
    fake.lib.fake_capture(None)
    (captured,) = launches(fake.log(), "megakernel")
    assert captured[1] not in work[0].values()
    with fake.failing_above(0):
        d.render(100, 60, 1, 0x9000)
    lines = fake.log()
    assert launches(lines, "megakernel") and not any(x.startswith("bad") for x in lines)


@pytest.mark.parametrize("scene,closest,any_hit", [
    # the ray counts up to which the lock-step kernels answer, in thousands; None: at any size
    (SPHERES_24, None, None), (FIELD, None, None), (REF_ROOM, None, None), ((15, 0), None, None),
    (SPHERES_488, 340, 1000), ((10, 2000), 227, 680), ((11, 2), 227, 227), (ROOM_1K, 227, 227), (ROOM_80K, 227, 227),
    ((12, 60), 340, 680), (INSTANCES, 227, 680), ((12, 2000), 227, 340), ((14, 0), 227, 568)])
def test_which_ray_queries_stream(fake, scene, closest, any_hit):
    """Closest and any hits take the kernel that was measured faster for that many rays in scenes like these."""
    d = DeviceScene(*scene)
    fake.log()
    for query, line in (("closest", closest), ("any", any_hit)):
        fn = getattr(fake.lib, f"pt_trace_{query}_device")
        for n in (1000, 120000, (line or 2500) * 1000 - 2000, (line or 2500) * 1000 + 25000, 16000000):
            assert fn(d.s.handle, SOME, n, 0.001, 1000.0, SOME, None) == 0
            form = "stream" if line and n > line * 1000 else "lock-step"
            assert fake.log() == [f"{query} {form}"], n


@pytest.mark.parametrize("scenes,streams", [
    # (scene, frame's width and height, samples, bounces), as often as given
    ([(SPHERES_24, 256, 2, 10)] * 8, False), ([(SPHERES_24, 512, 8, 10)] * 4, False),
    ([(SPHERES_24, 128, 3, 10)] * 8, True), ([((10, 2000), 256, 2, 10)] * 8, False),
    ([((10, 2000), 256, 3, 10)] * 8, True), ([(ROOM_1K, 256, 2, 10)] * 8, True), ([(ROOM_1K, 512, 4, 2)] * 4, False),
    ([((14, 0), 256, 2, 10)] * 8, False), ([((14, 0), 256, 4, 10)] * 8, True),
    ([(SPHERES_24, 512, 8, 10)] * 3 + [(ROOM_1K, 512, 8, 10)], True), ([(ROOM_1K, 128, 4, 10)] * 3, False),
    ([(ROOM_1K, 256, 2, 0)] * 8, False)])
def test_which_batches_stream(fake, scenes, streams):
    """Batches take the form that was measured faster for scenes like theirs."""
    import photon_tracer_b200 as pt
    items = []
    for k, ((kind, param), side, spp, _) in enumerate(scenes):
        g = pt.Generated(kind, seed=k + 1, param=param)
        items.append((g, g.camera, side, side, spp, k))
    b = pt.Batch(items, ONE_LAUNCH, max_bounces=scenes[0][3])
    assert one_launch_lines(fake, b) == ["batch stream" if streams else "batch 128"]
    b.close()


def test_gradients_that_the_tensor_cores_refuse_run_on_the_cuda_cores(fake):
    from photon_tracer_b200 import abi
    net = C.c_void_p()
    abi.check(fake.lib.pt_unet_create(1, C.byref(net)))
    fake.log()
    fake.lib.fake_tensor_cores(0)
    assert grads(fake, net, 1, 32, 48) == abi.PT_OK
    fake.lib.fake_tensor_cores(1)
    lines = fake.log()
    fake.lib.pt_unet_destroy(net)
    assert lines.count("wgrad") == 15 and lines.count("relu_grad") == 14
    assert not [x for x in lines if x.startswith("bad") or x.endswith("tc")]


def test_small_host_renders_keep_a_buffer_of_their_scene(fake):
    """A scanline's samples go through the scene's own buffer, which grows and goes with the scene; larger host frames
    take the pool's memory, as every frame on a caller's stream does."""
    import numpy as np
    import photon_tracer_b200 as pt
    before = fake.live_bytes()
    d = DeviceScene(SPHERES, 20)
    fake.log()
    for width, spp in ((400, 16), (1920, 40), (64, 4)):
        pt.render_row_linear(d.s, d.g.camera, 3, width, 200, spp, 10, np.empty((width, 3), np.float32), 1)
        lines = fake.log()
        assert len(launches(lines, "samples")) == 1 and not any(x.startswith("bad") for x in lines)
        assert f"malloc {256 + 12 * width * spp}" in lines or width == 64
    d.s.render(d.g.camera, 400, 225, 16)
    assert f"malloc {32 << 20}" in fake.log()
    d.render(64, 48, 4, 0x7000)
    assert f"malloc {1 << 20}" in fake.log()
    d.s.close()
    assert fake.live_bytes() == before


def test_gpu_comparisons_of_the_two_forms_have_both(fake):
    """Every frame that the GPU tests compare between the streaming form and a capture's lock-step form streams when it
    is not captured."""
    import test_gpu_stream
    import test_gpu_stream_forms
    import photon_tracer_b200 as pt
    (cases,) = [m.args[1] for m in test_gpu_stream.test_frames_equal_lock_step.pytestmark if m.name == "parametrize"]
    for kind, param, width, height, spp, depth, aux, flags, snapshot in cases + test_gpu_stream_forms.FORMS:
        g = pt.Generated(kind, seed=3, param=param)
        s = pt.Scene(g)
        st = s.settings(width, height, spp, depth, seed=9, flags=flags, rng=int(snapshot), states_ptr=64)
        fake.log()
        s.render_device(g.camera, st, SOME.value, SOME.value if aux else 0, 0, 0x7000)
        assert launches(fake.log(), "samples"), (kind, param, width, height, spp)
