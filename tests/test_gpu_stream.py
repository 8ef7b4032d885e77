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
