"""The library's host code over a stand-in for the CUDA runtime (fake_cudart.cpp): what is launched, captured, copied and
refused, without a GPU."""
from __future__ import annotations

import ctypes as C
import os
import subprocess

from multigridsoftbody_b200 import _lib as L
from multigridsoftbody_b200 import build

HERE = os.path.dirname(os.path.abspath(__file__))
CAPTURES, GRAPH_LAUNCHES, SYNCHRONISATIONS, UPLOADED, PINNED, ALLOCATED = range(6)


def build_host_only(out_dir: str) -> str:
    """The library's own objects linked against the stand-in instead of the CUDA runtime."""
    build.build_library()
    objs = [os.path.join(build.PKG, "_build", s + ".o") for s in build.SOURCES]
    sources = [os.path.join(build.CSRC, f) for f in os.listdir(build.CSRC)]
    if any(build._stale(o, sources) for o in objs):
        build.build_library(force=True)
    include = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(build._nvcc()))), "include")
    out = os.path.join(out_dir, "libmgsb_host.so")
    subprocess.run(["g++", "-O1", "-shared", "-fPIC", "-Wl,-Bsymbolic", "-I" + include, "-o", out,
                    os.path.join(HERE, "fake_cudart.cpp"), *objs], check=True)
    return out


class Host:
    """The loaded library and what its runtime wrote down."""

    def __init__(self, path: str):
        self.lib = C.CDLL(path)
        for name, res, args in L.SIGNATURES:
            fn = getattr(self.lib, name)
            fn.restype = res
            fn.argtypes = args
        self.lib.fake_count.restype = C.c_long

    def reset(self) -> None:
        self.lib.fake_reset()

    def refuse(self, kernel: str) -> None:
        self.lib.fake_refuse(kernel.encode())

    def count(self, what: int) -> int:
        return int(self.lib.fake_count(what))

    def launches(self, kernel: str = "") -> list[tuple]:
        """(kernel, grid, block, cluster, cooperative, shared memory) of the launches since the reset."""
        out, name, v = [], C.create_string_buffer(512), (C.c_ulonglong * 5)()
        for k in range(self.lib.fake_launches()):
            self.lib.fake_launch(k, name, 512, v)
            if kernel in name.value.decode():
                out.append((name.value.decode(), *(int(x) for x in v)))
        return out
