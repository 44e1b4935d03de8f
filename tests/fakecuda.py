"""libswave's host code on the CPU: the library's objects linked with
fake_cuda.cpp in place of the CUDA runtime.  Kernels do nothing, so results
mean nothing; what is launched, allocated and returned does."""
from __future__ import annotations

import contextlib
import ctypes as C
import os
import subprocess

import seismic_gb300 as sw
from seismic_gb300 import build

HERE = os.path.dirname(os.path.abspath(__file__))
SRC = os.path.join(HERE, "fake_cuda.cpp")
LIB = os.path.join(build.OBJDIR, "libswave_fake.so")


def _build() -> str:
    build.build_library()
    objs = [os.path.join(build.OBJDIR, s.replace(".cu", ".o")) for s in build.CUDA_SOURCES]
    if build._stale(LIB, [SRC, *objs]):
        inc = os.path.join(os.path.dirname(os.path.dirname(build._nvcc())), "include")
        obj, tmp = LIB + ".fake.o", LIB + ".new"
        for cmd in (["g++", "-O1", "-std=c++17", "-fPIC", "-I", inc, "-I",
                     os.path.join(build.ROOT, "include"), "-c", SRC, "-o", obj],
                    ["g++", "-shared", "-Wl,-Bsymbolic", "-Wl,--no-undefined", "-o", tmp, obj,
                     *objs]):
            r = subprocess.run(cmd, capture_output=True, text=True)
            assert r.returncode == 0, r.stderr
        os.replace(tmp, LIB)     # never over a mapped library
    return LIB


class Fake:
    """The fake's controls, and contexts of the library linked with it."""

    def __init__(self):
        self.lib = sw.load_library(_build())
        for name, res, args in (("fake_reset", None, [C.c_size_t]),
                                ("fake_fail_alloc", None, [C.c_int]),
                                ("fake_blocks_per_sm", None, [C.c_int]),
                                ("fake_coop_error", None, [C.c_int]),
                                ("fake_stale", C.c_int, []), ("fake_used", C.c_size_t, []),
                                ("fake_set_epoch", None, [C.c_void_p, C.c_uint]),
                                ("fake_epoch", C.c_uint, [C.c_void_p]),
                                ("fake_launches", C.c_char_p, [])):
            f = getattr(self.lib, name)
            f.restype, f.argtypes = res, args

    def reset(self, mem: int = 8 << 30):
        self.lib.fake_reset(mem)

    @contextlib.contextmanager
    def context(self):
        real, sw._lib = sw._lib, self.lib
        try:
            c = sw.Context(0)
        finally:
            sw._lib = real
        try:
            yield c
        finally:
            c.close()

    def launches(self) -> list[tuple[str, tuple[int, int, int], bool]]:
        """(kernel, grid, cooperative) in order; a captured launch appears once."""
        out = []
        for ln in self.lib.fake_launches().decode().splitlines():
            name, x, y, z, coop = ln.rsplit(" ", 4)
            out.append((name, (int(x), int(y), int(z)), coop == "1"))
        return out

    def kernels(self, part: str) -> list[tuple[str, tuple[int, int, int], bool]]:
        return [k for k in self.launches() if part in k[0]]
