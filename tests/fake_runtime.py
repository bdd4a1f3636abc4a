"""The library's host code on a stand-in for the CUDA runtime
(fake_cudart.cpp): no GPU, kernels do not run, device memory reads as zeros."""
import ctypes as C
import functools
import importlib.util
import os
import shutil
import subprocess
import tempfile

import numpy as np

import build as lib_build
import cipc

HERE = os.path.dirname(os.path.abspath(__file__))


class FakeRuntime:
    def __init__(self, path, sms):
        spec = importlib.util.spec_from_file_location("cipc_on_fake_runtime", cipc.__file__)
        self.cipc = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(self.cipc)
        self.cipc.LIB_PATH = path
        self.L = self.cipc.lib()
        self.L.fake_events.restype = C.c_char_p
        self.L.fake_device(sms)

    def reset(self):
        self.L.fake_reset()

    def events(self, kind, text=""):
        """The recorded events of a kind ("launch", "unordered", ...) whose line holds `text`."""
        return [e for e in self.L.fake_events().decode().splitlines() if e.startswith(kind + " ") and text in e]


@functools.lru_cache(None)
def _library():
    lib_build.build()
    objs = [os.path.join(lib_build.OUT, n + ".o") for n in list(lib_build.UNITS) + list(lib_build.HOST_UNITS)]
    tmp = tempfile.mkdtemp()
    so, harness = os.path.join(tmp, "libcipc_fake_runtime.so"), os.path.join(tmp, "device_buffer_harness.o")
    subprocess.run([lib_build.NVCC, *lib_build.ARCH, *lib_build.COMMON, "-c", os.path.join(HERE, "device_buffer_harness.cu"), "-o", harness], check=True)
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-Wl,-Bsymbolic", "-Wl,-z,defs", "-I/usr/local/cuda/include",
                    os.path.join(HERE, "fake_cudart.cpp"), harness, *objs, "-o", so, "-lpthread", "-ldl", "-lrt"], check=True)
    return so


@functools.lru_cache(None)
def runtime(sms=148):
    """The library on a device of `sms` multiprocessors (a copy of its own: the
    library asks for the count once)."""
    so = _library()
    return FakeRuntime(shutil.copy(so, so.replace(".so", "_%d.so" % sms)), sms)


def ring_system(nv, neighbours=(1, 2, 5)):
    """Block-CSR arrays of a ring of `nv` rows joined to the rows at the given
    distances (the values do not matter: kernels do not run)."""
    i = np.arange(nv)
    pairs = np.concatenate([np.stack([i, (i + d) % nv]) for d in (0,) + tuple(neighbours) + tuple(-d for d in neighbours)], axis=1)
    return _blocks(nv, pairs)


def hub_system(nv, every, degree):
    """As ring_system, a ring with every `every`-th row joined to `degree` others of them."""
    i = np.arange(nv)
    h = i[::every]
    to = [np.stack([i, (i + d) % nv]) for d in (0, 1, -1)]
    to += [np.stack([h, np.roll(h, d)]) for k in range(1, degree // 2 + 1) for d in (k, -k)]
    return _blocks(nv, np.concatenate(to, axis=1))


def _blocks(nv, pairs):
    key = np.unique(pairs[0].astype(np.int64) * nv + pairs[1])
    rp = np.concatenate([[0], np.cumsum(np.bincount(key // nv, minlength=nv))]).astype(np.int32)
    return rp, (key % nv).astype(np.int32), np.zeros((len(key), 3, 3)), np.zeros(3 * nv)
