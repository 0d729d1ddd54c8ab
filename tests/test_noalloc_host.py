"""iwpp_reconstruct_noalloc's host side, on the CPU: the library's own objects
linked against a stand-in for the CUDA runtime (native/noalloc_runtime.cpp)
that reports what it is told and records which kernels are loaded when."""
import ctypes
import os
import subprocess

import pytest

from iwpp import _build

HERE = os.path.join(os.path.dirname(os.path.abspath(__file__)), "native")
DEV_OK, DEV_ERR_TIMEOUT, DEV_ERR_OVERFLOW, DEV_ERR_INTERNAL = 0, 3, 5, 9
OK, ERR_TIMEOUT, ERR_OVERFLOW, ERR_INTERNAL = 0, 3, 5, 9


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    _build.build_iwpp()
    tmp = tmp_path_factory.mktemp("noalloc")
    layout, so = str(tmp / "layout.o"), str(tmp / "noalloc.so")
    subprocess.run([_build._nvcc(), *_build.NVCC_FLAGS, "-I" + _build.SRC_DIR, "-c",
                    os.path.join(HERE, "noalloc_layout.cu"), "-o", layout], check=True)
    objs = [os.path.join(_build.LIB_DIR, "obj", n + ".o")
            for n in ("iwpp_noalloc", "iwpp_engine", "iwpp_engine_async", "iwpp_engine_mutex", "iwpp_engine_double",
                      "iwpp_engine_unique")]
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(_build._nvcc())))
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-I" + os.path.join(cuda, "include"), "-o", so,
                    os.path.join(HERE, "noalloc_runtime.cpp"), layout, *objs, "-Wl,-Bsymbolic"], check=True)
    dll = ctypes.CDLL(so)
    fn = dll.iwpp_reconstruct_noalloc
    fn.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_size_t, ctypes.c_size_t] + [ctypes.c_int] * 4 + [
        ctypes.c_void_p]
    return dll


def _call(lib, w, h, conn, error=DEV_OK):
    """One call on a w x h uint8 image (its pointers are not followed here)."""
    lib.fake_reset(error)
    pitch = -(-w // 4) * 4
    return lib.iwpp_reconstruct_noalloc(256, 512, pitch, pitch, w, h, 0, conn, None)


@pytest.mark.parametrize("device_error, status", [(DEV_OK, OK), (DEV_ERR_TIMEOUT, ERR_TIMEOUT),
                                                  (DEV_ERR_OVERFLOW, ERR_OVERFLOW), (DEV_ERR_INTERNAL, ERR_INTERNAL)])
def test_a_failed_job_is_no_success(lib, device_error, status):
    assert _call(lib, 300, 200, 8, device_error) == status


def test_the_first_call_loads_every_kernel(lib):
    # A kernel that a later call is the first to launch is loaded then, which
    # may take device memory and wait for the device.
    assert _call(lib, 300, 200, 8) == OK
    loads = ctypes.c_int.in_dll(lib, "fake_launches_that_load")
    loaded = lib.fake_loaded()
    kernels = 0
    for conn in (4, 8):
        for w, h in ((300, 200), (4096, 2112), (4224, 4037), (32768, 20000)):
            before = loads.value
            assert _call(lib, w, h, conn) == OK
            assert lib.fake_launches() == 1
            assert (loads.value, lib.fake_loaded()) == (before, loaded), (conn, w, h)
            kernels += 1
    assert kernels == 8
