"""The library's host code over a fake CUDA runtime (fake_cuda.cpp): builds
both into one shared library and puts it in the place of libphoton_cuda.so."""
import concurrent.futures as cf
import contextlib
import ctypes as C
import os
import subprocess

from conftest import ROOT


def build_fake(out_dir):
    from photon_tracer_b200.build import CSRC, CXX_FLAGS
    sources = [os.path.join(CSRC, f) for f in sorted(os.listdir(CSRC)) if f.endswith(".cpp")]
    sources.append(os.path.join(ROOT, "tests", "fake_cuda.cpp"))
    objects = [os.path.join(out_dir, os.path.basename(s) + ".o") for s in sources]

    def run(cmd):
        res = subprocess.run(cmd, capture_output=True, text=True)
        assert res.returncode == 0, res.stderr

    flags = [f for f in CXX_FLAGS if f != "-O2"] + ["-O1"]
    with cf.ThreadPoolExecutor(8) as ex:
        list(ex.map(lambda so: run(["g++"] + flags + ["-c", so[0], "-o", so[1]]), zip(sources, objects)))
    path = os.path.join(out_dir, "libfake.so")
    # its own runtime, also where a process has the real one loaded
    run(["g++", "-shared", "-Wl,-Bsymbolic", "-o", path] + objects + ["-lpthread"])
    return path


class Fake:
    """The test's side of the fake runtime."""

    def __init__(self, path):
        from photon_tracer_b200 import abi
        self.lib = C.CDLL(path)
        for name, res, args in abi.PROTOTYPES:
            if hasattr(self.lib, name):
                fn = getattr(self.lib, name)
                fn.restype, fn.argtypes = res, args
        self.lib.fake_log.restype = C.c_char_p
        self.lib.fake_live_bytes.restype = C.c_size_t
        self.lib.fake_fail_after.argtypes = [C.c_long]
        self.lib.fake_fail_above.argtypes = [C.c_size_t]
        self.lib.fake_budget.argtypes = [C.c_size_t]
        self.lib.fake_capture.argtypes = [C.c_void_p]

    def log(self):
        """The events since the last call."""
        lines = self.lib.fake_log().decode().splitlines()
        self.lib.fake_clear()
        return lines

    def live_bytes(self):
        return self.lib.fake_live_bytes()

    def fail_after(self, n):
        """The next n device allocations succeed and the ones after them fail; -1: none fails."""
        self.lib.fake_fail_after(n)

    @contextlib.contextmanager
    def failing_above(self, n_bytes):
        self.lib.fake_fail_above(n_bytes)
        try:
            yield
        finally:
            self.lib.fake_fail_above(2**64 - 1)

    @contextlib.contextmanager
    def budget(self, n_bytes):
        """Device memory for n_bytes in all."""
        self.lib.fake_budget(n_bytes)
        try:
            yield
        finally:
            self.lib.fake_budget(2**64 - 1)

    @contextlib.contextmanager
    def falling_times(self):
        """Events measure less time from call to call, so that the last of several candidates is the fastest."""
        self.lib.fake_falling_times(1)
        try:
            yield
        finally:
            self.lib.fake_falling_times(0)
