"""The streaming tree walks against the oracle at the sizes where their hand-out
of rays can go wrong (the first count that streams on 148 SMs, runs that end
inside a warp, warps with unequal runs), on flat and two-level trees, with leaves up to the 15
primitives that a stack word holds and beyond them (the lock-step walk)."""
import numpy as np
import pytest

from handmade import scene_from, tri
from test_gpu_trace import assert_hits_equal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,param,extent", [(10, 0, 6.0), (11, 3, 1.0), (12, 60, 60.0)])
@pytest.mark.parametrize("n", [227329, 227360, 341001])
def test_ray_counts(built, kind, param, extent, n):
    from oracle.oracle import Oracle
    g = built.Generated(kind, seed=4, param=param)
    s, o = built.Scene(g), Oracle(g.desc)
    rays = built.generate_rays(n, [-extent] * 3, [extent] * 3, n)
    assert_hits_equal(s.trace_closest(rays), o.trace_closest(rays, threads=8), rays)
    assert np.array_equal(s.trace_any(rays, 0.001, extent), o.trace_any(rays, 0.001, extent))


@pytest.mark.parametrize("copies", [1, 8, 15, 16, 40])
def test_leaf_sizes(built, copies):
    """Coincident triangles cannot be split: one leaf holds them all."""
    from oracle.oracle import Oracle
    from photon_tracer_b200 import abi
    m = [abi.pt_material(type=0, albedo=abi.F3(0.5, 0.5, 0.5))]
    tris = [tri(built, (-1, -1, 0), (1, -1, 0), (0, 1, 0)) for _ in range(copies)]
    tris += [tri(built, (x, -1, -1), (x + 0.5, -1, -1), (x, 1, -1)) for x in np.linspace(-2, 2, 20)]
    d = scene_from(built, m, [abi.pt_sphere(center=abi.F3(0, 0, -2), radius=0.5)], tris)
    s, o = built.Scene(d.desc_ptr), Oracle(d.desc)
    rng, n = np.random.default_rng(copies), 240000
    rays = np.concatenate([rng.uniform(-1, 1, (n, 2)), np.full((n, 1), 2.0), rng.normal(0, 0.3, (n, 2)),
                           np.full((n, 1), -1.0)], 1).astype(np.float32)
    assert_hits_equal(s.trace_closest(rays), o.trace_closest(rays, threads=8), rays)
    assert np.array_equal(s.trace_any(rays), o.trace_any(rays))


def _frame(torch, scene, cam, st, aux):
    out = torch.full((st.height, st.width, 3), float("nan"), device="cuda")
    ax = torch.full((st.height, st.width, 7), float("nan"), device="cuda") if aux else None
    rays = torch.zeros(1, dtype=torch.int64, device="cuda")
    return out, ax, rays, lambda: scene.render_device(cam, st, out.data_ptr(), ax.data_ptr() if aux else 0,
                                                      rays.data_ptr(), torch.cuda.current_stream().cuda_stream)


@pytest.mark.parametrize("kind,param,width,height,spp,depth,aux,flags,snapshot", [
    (10, 0, 2, 2, 4, 10, False, 0, False),          # fewer samples than warps
    (10, 40, 33, 17, 5, 10, True, 0, False),        # tiles past the right and lower edge
    (11, 3, 65, 3, 7, 1, True, 0, False),           # one bounce; fewer rows than a tile
    (11, 3, 200, 113, 2, 10, False, 0, True),       # caller's random states
    (11, 2, 1024, 1024, 24, 4, False, 0, False),    # more samples than one launch's buffer holds
    (11, 2, 640, 360, 40, 3, True, 0, False),       # the same with auxiliary outputs
    (12, 200, 97, 61, 6, 10, True, 0, False),
    (14, 0, 97, 61, 6, 10, True, 0, False),         # textures, with instances
    (15, 0, 97, 61, 6, 10, True, 1, False),         # extended light sampling
    (15, 0, 97, 61, 6, 10, False, 1, False),
])
def test_frames_equal_lock_step(built, kind, param, width, height, spp, depth, aux, flags, snapshot):
    """A captured render cannot keep a sample buffer and takes the lock-step
    form; the image, the guides and the ray count are the same bit for bit."""
    import torch
    from photon_tracer_b200 import abi
    g = built.Generated(kind, seed=3, param=param)
    s = built.Scene(g)
    states = None
    if snapshot:
        gen = torch.Generator(device="cuda").manual_seed(5)
        states = torch.randint(-2**62, 2**62, (width * height * spp, 4), device="cuda", generator=gen)
    st = built.Scene.settings(width, height, spp, depth, seed=9, first_sample=3, flags=flags,
                              rng=abi.PT_RNG_SNAPSHOT if snapshot else abi.PT_RNG_SAMPLE,
                              states_ptr=states.data_ptr() if snapshot else None)
    out, ax, rays, render = _frame(torch, s, g.camera, st, aux)
    render()
    s.sync(torch.cuda.current_stream().cuda_stream)
    out2, ax2, rays2, render2 = _frame(torch, s, g.camera, st, aux)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        render2()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.isfinite(out).all()
    assert torch.equal(out.view(torch.int32), out2.view(torch.int32))
    assert int(rays) == int(rays2) > 0
    if aux:
        assert torch.equal(ax.view(torch.int32), ax2.view(torch.int32))


@pytest.mark.parametrize("sizes", [
    [(2, 2, 70000), (33, 17, 500)],              # more samples of a pixel than a launch of one scene needs
    [(640, 361, 64), (200, 3, 3), (500, 333, 120), (31, 65, 1)],  # launches that end inside a scene
])
def test_streamed_batch(built, sizes):
    """A batch large enough to stream gives each scene the image its own
    render gives, whatever launch its samples fall into."""
    from photon_tracer_b200 import abi
    items = []
    for k, (w, h, spp) in enumerate(sizes):
        g = built.Generated([11, 10, 12][k % 3], seed=k + 1, param=[2, 30, 60][k % 3])
        items.append((g, g.camera, w, h, spp, 50 + k))
    b = built.Batch(items, abi.PT_BATCH_ONE_LAUNCH, max_bounces=3)
    for _ in range(2):
        rays, total = b.render(), 0
        for i, (g, cam, w, h, spp, seed) in enumerate(items):
            img, _, r = built.Scene(g).render(cam, w, h, spp, 3, seed=seed)
            total += r
            assert b.image(i).tobytes() == img.tobytes(), f"scene {i}"
        assert rays == total
    times = b.scene_times()
    assert np.all(times > 0) and np.all(np.isfinite(times))


@pytest.mark.parametrize("kind,param,extent,n", [(10, 0, 6.0, 1023011), (12, 60, 60.0, 682017), (14, 0, 1.0, 568353)])
def test_any_hit_ray_counts(built, kind, param, extent, n):
    """Any hits of open and of instanced scenes stream from larger counts on."""
    from oracle.oracle import Oracle
    g = built.Generated(kind, seed=4, param=param)
    rays = built.generate_rays(n, [-extent] * 3, [extent] * 3, n)
    s, o = built.Scene(g), Oracle(g.desc)
    assert np.array_equal(s.trace_any(rays, 0.001, extent), o.trace_any(rays, 0.001, extent))


@pytest.mark.parametrize("copies", [8, 15, 16])
def test_leaf_sizes_of_a_scene_that_streams(built, copies):
    """As test_leaf_sizes, among enough other triangles for its trees to be walked as streams."""
    from oracle.oracle import Oracle
    from photon_tracer_b200 import abi
    m = [abi.pt_material(type=0, albedo=abi.F3(0.5, 0.5, 0.5))]
    tris = [tri(built, (-1, -1, 0), (1, -1, 0), (0, 1, 0)) for _ in range(copies)]
    tris += [tri(built, (x, y, -1), (x + 0.1, y, -1), (x, y + 0.1, -1.2)) for x in np.linspace(-2, 2, 25)
             for y in np.linspace(-2, 2, 20)]
    d = scene_from(built, m, [abi.pt_sphere(center=abi.F3(0, 0, -2), radius=0.5)], tris)
    s, o = built.Scene(d.desc_ptr), Oracle(d.desc)
    assert 128 * s.info().n_nodes + 48 * s.info().n_slots > 16 << 10
    rng, n = np.random.default_rng(copies), 240000
    rays = np.concatenate([rng.uniform(-1, 1, (n, 2)), np.full((n, 1), 2.0), rng.normal(0, 0.3, (n, 2)),
                           np.full((n, 1), -1.0)], 1).astype(np.float32)
    assert_hits_equal(s.trace_closest(rays), o.trace_closest(rays, threads=8), rays)
    assert np.array_equal(s.trace_any(rays), o.trace_any(rays))
