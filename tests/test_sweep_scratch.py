"""Scratch that the whole-image sweeps ask for: where they go through kernels
that use it, and nowhere else (the library's own objects on the CPU, linked
against the stand-in for the CUDA runtime)."""
import ctypes
import os
import subprocess

import pytest

from iwpp import _build

HERE = os.path.join(os.path.dirname(os.path.abspath(__file__)), "native")


@pytest.fixture(scope="module")
def scratch_bytes(tmp_path_factory):
    _build.build_iwpp()
    tmp = tmp_path_factory.mktemp("sweeps")
    objs, so = [str(tmp / "scratch.o"), str(tmp / "layout.o")], str(tmp / "sweeps.so")
    for src, obj in zip(("sweep_scratch.cu", "noalloc_layout.cu"), objs):
        subprocess.run([_build._nvcc(), *_build.NVCC_FLAGS, "-I" + _build.SRC_DIR, "-c", os.path.join(HERE, src),
                        "-o", obj], check=True)
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(_build._nvcc())))
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-I" + os.path.join(cuda, "include"), "-o", so,
                    os.path.join(HERE, "noalloc_runtime.cpp"), *objs,
                    os.path.join(_build.LIB_DIR, "obj", "iwpp_sweeps.o"), "-Wl,-Bsymbolic"], check=True)
    fn = ctypes.CDLL(so).scratch_bytes
    fn.argtypes = [ctypes.c_size_t, ctypes.c_size_t, ctypes.c_longlong] + [ctypes.c_int] * 4
    fn.restype = ctypes.c_size_t

    def call(w, h, dt, conn, pitch=None, base=256):
        pitch = pitch or -(-w * (1, 2, 4)[dt] // 4) * 4
        return fn(base, 1 << 30, pitch, w, h, dt, conn)

    return call


def test_only_the_segmented_sweeps_have_scratch(scratch_bytes):
    assert scratch_bytes(4096, 4096, 0, 4) == 3 * 4 * 64 * 32 * 4  # four segments, 64 strips of 64 bytes
    assert scratch_bytes(2048, 4096, 1, 4) == 3 * 4 * 64 * 32 * 4
    for args in ((4096, 2048, 0, 4), (4096, 4096, 0, 8), (4096, 4096, 2, 4)):
        assert scratch_bytes(*args) == 0, args


@pytest.mark.parametrize("w, dt, pitch, base", [(4100, 0, None, 256), (4095, 0, 4096, 256), (2050, 1, None, 256),
                                                (4096, 0, 4100, 256), (4096, 0, None, 260)])
def test_sweeps_by_strips_have_none(scratch_bytes, w, dt, pitch, base):
    # rows that are not whole strips, or off the 16-byte boundary
    assert scratch_bytes(w, 4096, dt, 4, pitch, base) == 0
