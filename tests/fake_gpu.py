"""The library's own objects linked with a CUDA runtime that runs nothing
(host_harness/fake_cudart.cpp), so that its host code - what it allocates,
launches and reports - is tested without a GPU."""
import contextlib
import ctypes as C
import glob
import os
import shutil
import subprocess
import tempfile
from dataclasses import dataclass

import common
import torch_b200

_path = None


def library():
    """Path of the library with the fake runtime (linked once per process)."""
    global _path
    if _path is None:
        subprocess.run(["make", "-s", "-C", os.path.join(common.ROOT, "torch_b200", "csrc")], check=True)
        d = tempfile.mkdtemp(prefix="fake_gpu_")
        _path = os.path.join(d, "libtorch_b200_fake.so")
        nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
        inc = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
        objs = sorted(glob.glob(os.path.join(common.ROOT, "_build", "torch_b200", "*.o")))
        subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-Wl,-Bsymbolic", "-I", inc, "-o", _path,
                        os.path.join(common.HERE, "host_harness", "fake_cudart.cpp"), *objs], check=True)
    return _path


@dataclass
class Launch:
    name: str
    grid: int
    block: int
    smem: int
    programmatic: int


class Gpu:
    def __init__(self, lib):
        self.lib = lib
        lib.fake_launches.restype = lib.fake_most_smem_settings.restype = C.c_longlong
        lib.fake_launch.restype = C.c_char_p
        lib.fake_launch.argtypes = [C.c_longlong, C.c_void_p]
        lib.fake_refuse.argtypes = [C.c_char_p]

    def reset(self):
        self.lib.fake_reset()

    def refuse(self, part):
        self.lib.fake_refuse(part.encode())

    def counts(self):
        v = (C.c_longlong * 5)()
        self.lib.fake_counts(v)
        return dict(zip(("allocations", "live", "synchronisations", "refused", "graphs"), v))

    def launches(self):
        out = []
        for i in range(self.lib.fake_launches()):
            v = (C.c_longlong * 4)()
            name = self.lib.fake_launch(i, v).decode()
            out.append(Launch(name, *v))
        return out

    def most_smem_settings(self):
        return int(self.lib.fake_most_smem_settings())


@contextlib.contextmanager
def fake_gpu():
    """torch_b200 on the fake runtime while the context is open."""
    saved = torch_b200._lib, torch_b200.library_path
    torch_b200._lib, torch_b200.library_path = None, library
    try:
        gpu = Gpu(torch_b200.load_library())
        gpu.reset()
        yield gpu
    finally:
        torch_b200._lib, torch_b200.library_path = saved
