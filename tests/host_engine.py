"""The engine's host code on a fake CUDA runtime (fake_cudart.cpp), for tests of
the order and outcome of its runtime calls without a GPU.  Kernels do not run:
device memory reads as zeros."""
import contextlib
import ctypes
import gc
import os
import shutil
import subprocess

import pytest

import riskgpu
from riskgpu import build

HERE = os.path.dirname(os.path.abspath(__file__))
OOM = 2  # cudaErrorMemoryAllocation


def link(folder):
    """One shared library of the engine's objects and the fake runtime."""
    build.build()
    include = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(build._nvcc()))), "include")
    if not os.path.exists(os.path.join(include, "cuda_runtime_api.h")):
        include = "/usr/local/cuda/include"
    out = os.path.join(folder, "libriskgpu_host.so")
    objects = [os.path.join(build.OUT, os.path.basename(c)[:-3] + ".o") for c in build._sources()[0]]
    subprocess.run(["g++", "-std=c++17", "-O1", "-fPIC", "-shared", "-Wl,-Bsymbolic", "-I" + include, "-o", out,
                    os.path.join(HERE, "fake_cudart.cpp")] + objects, check=True)
    return out


class Fake:
    def __init__(self, lib):
        self.lib = lib
        for f in ("fake_log", "fake_live_bytes", "fake_peak_bytes"):
            getattr(lib, f).restype = ctypes.c_size_t

    def reset(self):
        self.lib.fake_reset()

    def log(self):
        """[(name, stream, detail)] since the last reset."""
        buf = ctypes.create_string_buffer(self.lib.fake_log(None, 0) + 1)
        self.lib.fake_log(buf, ctypes.c_size_t(len(buf)))
        return [tuple(line.split("|")) for line in buf.value.decode().splitlines()]

    def names(self):
        return [name for name, _, _ in self.log()]

    def fail(self, name, err, skip=0, count=1, until=None):
        self.lib.fake_fail(name.encode(), skip, count, err, until.encode() if until else None)

    def gather(self, name, count):
        self.lib.fake_gather(name.encode(), count)

    def free_bytes(self, *values):
        self.lib.fake_free_bytes((ctypes.c_size_t * len(values))(*values), len(values))

    def live(self):
        return self.lib.fake_live_bytes()

    def peak(self):
        return self.lib.fake_peak_bytes()


@contextlib.contextmanager
def engine(linked, folder):
    """riskgpu bound to a library of its own (fresh process-wide state)."""
    path = os.path.join(folder, "libriskgpu_fresh.so")
    shutil.copy(linked, path)
    was = riskgpu.LIB_PATH, riskgpu._lib
    riskgpu.LIB_PATH, riskgpu._lib = path, None
    try:
        yield Fake(riskgpu.lib())
    finally:
        for o in gc.get_objects():  # no handle of this library outlives its binding
            if isinstance(o, (riskgpu.Portfolio, riskgpu.Batch, riskgpu.Server)):
                o._h = ctypes.c_void_p()
        riskgpu.LIB_PATH, riskgpu._lib = was


# ---- fixtures (imported by the test files)
@pytest.fixture(scope="session")
def linked(tmp_path_factory):
    return link(str(tmp_path_factory.mktemp("linked")))


@pytest.fixture
def fake(linked, tmp_path, monkeypatch):
    monkeypatch.setenv("RG_TUNE_CACHE", str(tmp_path / "tune.json"))
    with engine(linked, str(tmp_path)) as f:
        yield f
