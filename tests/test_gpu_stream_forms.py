"""The streaming renders' forms that test_gpu_stream.py does not reach: one
sample per pixel, callers' random states with guides and over several launches,
extended light sampling among instances and with textures; and batches that
render scene by scene or choose how. As there, a captured render, which takes the
lock-step form, is the other side."""
import numpy as np
import pytest

from test_gpu_stream import test_frames_equal_lock_step as frames_equal_lock_step

pytestmark = pytest.mark.gpu

FORMS = [
    (11, 3, 1024, 1024, 1, 10, False, 0, False),   # one sample
    (11, 3, 1152, 1000, 1, 10, True, 0, False),
    (11, 3, 97, 61, 6, 10, True, 0, True),         # callers' states with guides
    (12, 60, 97, 61, 5, 10, True, 0, True),
    (11, 3, 1024, 1024, 24, 3, False, 0, True),    # over two launches
    (11, 3, 640, 640, 24, 3, True, 0, True),
    (12, 200, 97, 61, 6, 10, True, 1, False),      # extended light sampling
    (12, 200, 97, 61, 6, 10, False, 1, False),
    (14, 0, 97, 61, 6, 10, True, 1, False),
    (14, 0, 97, 61, 6, 10, False, 1, False),
    (14, 0, 97, 61, 6, 10, False, 0, True),
]


@pytest.mark.parametrize("kind,param,width,height,spp,depth,aux,flags,snapshot", FORMS)
def test_forms_equal_lock_step(built, kind, param, width, height, spp, depth, aux, flags, snapshot):
    frames_equal_lock_step(built, kind, param, width, height, spp, depth, aux, flags, snapshot)


@pytest.mark.parametrize("strategy", ["PER_SCENE_MEGA", "AUTO"])
def test_large_batch_scene_by_scene(built, strategy):
    """A batch whose scenes stream one by one, or in one launch or not as the autotuner finds, on two streams in turn:
    each scene's image is the one its own render gives."""
    import torch
    from photon_tracer_b200 import abi
    items = []
    for k, (w, h, spp) in enumerate([(640, 361, 16), (200, 97, 5), (500, 333, 24), (31, 65, 4)]):
        g = built.Generated([11, 10, 12, 14][k], seed=k + 1, param=[3, 300, 60, 0][k])
        items.append((g, g.camera, w, h, spp, 50 + k))
    b = built.Batch(items, getattr(abi, "PT_BATCH_" + strategy), max_bounces=4)
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    for k in range(4):
        b.render(stream=streams[k % 2].cuda_stream, count_rays=False)
    for i, (g, cam, w, h, spp, seed) in enumerate(items):
        img, _, _ = built.Scene(g).render(cam, w, h, spp, 4, seed=seed)
        assert b.image(i).tobytes() == img.tobytes(), f"scene {i}"
    assert np.all(np.isfinite(b.scene_times()))
