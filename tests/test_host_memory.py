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
