"""The a-trous passes at the sizes where their tiles can go wrong (one pixel,
images smaller than a tap's reach, one pixel past a tile in each direction),
with a scratch buffer that does not allow 16-byte accesses, and into the
caller's albedo buffer, against the oracle's filter."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,shift,into_albedo", [
    (1, 1, 0, False), (2, 33, 0, False), (32, 8, 0, False), (33, 9, 1, False), (31, 65, 0, True), (70, 41, 3, True),
    (257, 130, 0, False), (515, 7, 2, False)])
def test_atrous_sizes(built, w, h, shift, into_albedo):
    import torch
    from oracle.oracle import oracle_denoise
    from photon_tracer_b200 import abi
    rng = np.random.default_rng(w * 1000 + h)
    color = rng.gamma(1.0, 0.5, (h, w, 3)).astype(np.float32)
    albedo = rng.uniform(0, 1, (h, w, 3)).astype(np.float32).round(1)
    normal = rng.normal(0, 1, (h, w, 3)).astype(np.float32).round(0)
    normal[rng.uniform(size=(h, w)) < 0.2] = 0
    variance = rng.gamma(1.0, 0.1, (h, w)).astype(np.float32)
    want = oracle_denoise(color, albedo, normal, variance)
    d = [torch.from_numpy(a).cuda() for a in (color, albedo, normal, variance)]
    scratch = torch.empty(11 * w * h + shift, device="cuda")[shift:]
    out = d[1] if into_albedo else torch.empty((h, w, 3), device="cuda")
    ptr = lambda t: C.c_void_p(t.data_ptr())
    abi.check(built.load().pt_denoise_atrous_device(w, h, *[ptr(t) for t in d], ptr(out), ptr(scratch),
                                                    C.c_void_p(torch.cuda.current_stream().cuda_stream)))
    got = out.cpu().numpy()
    # expf may differ by an ulp, which the variance-scaled luminance weights of later passes amplify
    np.testing.assert_allclose(got, want, rtol=1e-3, atol=1e-5)


@pytest.mark.parametrize("at", [0.0, 1.5, 3.0, 4.0, 5.5, 6.0, 8.0])
def test_atrous_into_its_scratch(built, at):
    """The image may go into the scratch itself, at any place (floats per pixel from its start)."""
    import torch
    from photon_tracer_b200 import abi
    w, h = 70, 42
    gen = torch.Generator(device="cuda").manual_seed(7)
    d = [torch.rand((h, w) + s, device="cuda", generator=gen) for s in ((3,), (3,), (3,), ())]
    ptr = lambda t: C.c_void_p(t.data_ptr())
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    run = lambda out, scratch: abi.check(built.load().pt_denoise_atrous_device(
        w, h, *[ptr(t) for t in d], ptr(out), ptr(scratch), stream))
    want, scratch = torch.empty((h, w, 3), device="cuda"), torch.empty(11 * w * h, device="cuda")
    run(want, scratch)
    out = scratch[int(at * w * h):][:3 * w * h]
    run(out, scratch)
    assert torch.equal(out.view(h, w, 3), want)


@pytest.mark.parametrize("w,h,shift", [(1, 21000, 0), (16, 5003, 1), (33, 20001, 0), (20001, 3, 0), (47, 9001, 2)])
def test_atrous_strips(built, w, h, shift):
    """Narrow and flat images, whose wider passes go pixel by pixel."""
    import torch
    from oracle.oracle import oracle_denoise
    from photon_tracer_b200 import abi
    rng = np.random.default_rng(w)
    color = rng.gamma(1.0, 0.5, (h, w, 3)).astype(np.float32)
    albedo = rng.uniform(0, 1, (h, w, 3)).astype(np.float32).round(1)
    normal = rng.normal(0, 1, (h, w, 3)).astype(np.float32).round(0)
    normal[rng.uniform(size=(h, w)) < 0.2] = 0
    variance = rng.gamma(1.0, 0.1, (h, w)).astype(np.float32)
    want = oracle_denoise(color, albedo, normal, variance)
    d = [torch.from_numpy(a).cuda() for a in (color, albedo, normal, variance)]
    scratch, out = torch.empty(11 * w * h + shift, device="cuda")[shift:], torch.empty((h, w, 3), device="cuda")
    ptr = lambda t: C.c_void_p(t.data_ptr())
    abi.check(built.load().pt_denoise_atrous_device(w, h, *[ptr(t) for t in d], ptr(out), ptr(scratch),
                                                    C.c_void_p(torch.cuda.current_stream().cuda_stream)))
    np.testing.assert_allclose(out.cpu().numpy(), want, rtol=1e-3, atol=1e-5)  # as test_atrous_sizes
