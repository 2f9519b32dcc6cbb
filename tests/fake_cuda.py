"""The library linked to a CUDA runtime that only records (fake_cudart.cpp), for
tests of the host engine without a GPU: under the `rt` fixture genoaligner_gb300.api
calls a fresh copy of it, with host tensors for device memory, and rt.log() gives
the lines that runtime wrote."""
import contextlib
import ctypes
import os
import shutil
import subprocess

import pytest

from genoaligner_gb300 import _build, api

HERE = os.path.dirname(os.path.abspath(__file__))


def build(folder):
    """Links the library's objects with the fake runtime; the path."""
    _build.build()
    objs = [os.path.join(_build.OUT, s.rsplit(".", 1)[0] + ".o") for s in _build.SOURCES]
    if not all(os.path.exists(o) for o in objs):
        _build.build(force=True)
    out = os.path.join(str(folder), "libga_fake.so")
    include = os.path.join(os.path.dirname(os.path.dirname(_build.nvcc())), "include")
    subprocess.run(["g++", "-std=c++17", "-O1", "-fPIC", "-shared", "-Wl,-Bsymbolic", "-I" + include, "-o", out,
                    os.path.join(HERE, "fake_cudart.cpp"), *objs, "-lpthread"], check=True)
    return out


class Runtime:
    def __init__(self, lib):
        self.lib = lib
        lib.fake_log.restype = ctypes.c_char_p

    def clear(self):
        self.lib.fake_clear()

    def log(self):
        """The lines since the last clear()."""
        return self.lib.fake_log().decode().splitlines()

    def count(self, word):
        return sum(word in line for line in self.log())

    def stream(self, priority=0):
        s = ctypes.c_void_p()
        self.lib.cudaStreamCreateWithPriority(ctypes.byref(s), 0, priority)
        return s.value

    def capturing(self, stream, on):
        self.lib.fake_capturing(ctypes.c_void_p(stream), int(on))

    def set_device(self, d):
        self.lib.cudaSetDevice(d)


@contextlib.contextmanager
def library(path, folder):
    """api on a private copy of the library at `path` (its own contexts and graphs)."""
    copy = os.path.join(str(folder), "libga_fake_copy.so")
    shutil.copy(path, copy)
    kept, kept_build = api._lib, _build.build
    api._lib, _build.build = None, lambda *a, **k: copy
    try:
        yield Runtime(api.load())
    finally:
        api._lib, _build.build = kept, kept_build


@pytest.fixture(scope="module")
def fake_path(tmp_path_factory):
    return build(tmp_path_factory.mktemp("fake"))


@pytest.fixture
def rt(fake_path, tmp_path):
    with library(fake_path, tmp_path) as r:
        yield r
