"""The library's host side linked with fake_device.cpp instead of the CUDA
runtime and the kernels (no device needed)."""
import contextlib
import ctypes as C
import os
import subprocess
import tempfile

from anacapa_b200 import api, build

HERE = os.path.dirname(os.path.abspath(__file__))
HOST, DEVICE, MANAGED = 1, 2, 3  # cudaMemoryType
_dir = None


def _build():
    global _dir
    if _dir is None:
        _dir = tempfile.TemporaryDirectory(prefix="fake_device_")
        out = os.path.join(_dir.name, "libfake.so")
        src = [os.path.join(build.CSRC, f) for f in ("capi.cpp", "prepare.cpp", "staging.cpp", "film_io.cpp")]
        subprocess.run([os.environ.get("CXX", "g++"), "-O1", "-std=c++17", "-shared", "-fPIC", "-pthread",
                        "-ffp-contract=off", "-Wl,-Bsymbolic", f"-I{build.CUDA_HOME}/include", f"-I{build.ROOT}/include",
                        f"-I{build.CSRC}", *src, os.path.join(HERE, "fake_device.cpp"), "-o", out, "-lz"], check=True)
    return os.path.join(_dir.name, "libfake.so")


@contextlib.contextmanager
def fake_device(capacity=1 << 30):
    """api.* on the fake; yields the loaded library with the fake_* calls."""
    path, kept = _build(), (api._lib, api.LIB_PATH)
    api._lib, api.LIB_PATH = None, path
    try:
        L = api.lib()
        for name in ("fake_held", "fake_largest"):
            getattr(L, name).restype = C.c_size_t
        for name in ("fake_calls", "fake_direct_bytes", "fake_extend_rays", "fake_bad_records", "fake_good_records"):
            getattr(L, name).restype = C.c_long
        L.fake_reset.argtypes = [C.c_size_t]
        L.fake_fail.argtypes = [C.c_char_p, C.c_long, C.c_long]
        L.fake_calls.argtypes = [C.c_char_p]
        L.fake_mark.argtypes = [C.c_void_p, C.c_size_t, C.c_int]
        L.fake_fail_new.argtypes = [C.c_long]
        L.fake_reset(capacity)
        yield L
        assert L.fake_held() == 0, "device memory of closed contexts"
    finally:
        api._lib, api.LIB_PATH = kept
