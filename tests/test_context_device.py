"""A context's calls go to the context's device, whichever device is current (no GPU needed).

csrc/vt_api.cu is compiled against a host-only CUDA runtime with two devices (fake_cudart.cpp). Reading
an image back from one context while the other's device is current must wait for the first's device and
record its staging events there, for images small enough for one copy and for ones the threads drain.
"""
import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

from metal_vibe_tracer_b200 import build

HERE = Path(__file__).resolve().parent


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    tmp = tmp_path_factory.mktemp("fake")
    api, fake = tmp / "vt_api.o", tmp / "fake_cudart.o"
    include = ["-I", str(build.INCLUDE), "-I", str(build.CSRC)]
    subprocess.run([build.nvcc(), *build.ARCH, *build.NVCC_FLAGS, *include, "-c", str(build.CSRC / "vt_api.cu"), "-o", str(api)], check=True)
    cuda = Path(build.nvcc()).resolve().parent.parent / "include"
    subprocess.run(["g++", "-std=c++17", "-O1", "-fPIC", *include, "-I", str(cuda), "-c", str(HERE / "fake_cudart.cpp"), "-o", str(fake)],
                   check=True)
    out = tmp / "libvt_fake.so"
    subprocess.run(["g++", "-shared", "-pthread", "-Wl,-Bsymbolic", "-o", str(out), str(api), str(fake)], check=True)  # no CUDA runtime
    so = C.CDLL(str(out))
    so.fake_scene.restype = C.c_void_p
    so.fake_scene.argtypes = [C.c_int, C.c_uint32, C.c_uint32, C.c_uint32, C.c_double]
    so.vt_ctx_create.argtypes = [C.c_int32, C.c_void_p]
    so.vt_accum_readback.argtypes = [C.c_void_p, C.c_void_p, C.c_void_p, C.c_uint32, C.c_void_p]
    so.vt_last_error.restype, so.vt_last_error.argtypes = C.c_char_p, [C.c_void_p]
    return so


@pytest.mark.parametrize("size", [(16, 9), (640, 400)])
def test_readback_of_the_context_whose_device_is_not_current(lib, size):
    w, h = size
    ctx = [C.c_void_p(), C.c_void_p()]
    for d in (0, 1):
        assert lib.vt_ctx_create(d, C.byref(ctx[d])) == 0
    for d in (0, 1, 0):  # the call before left the other device current
        lib.cudaSetDevice(1 - d)
        scene = lib.fake_scene(d, w, h, 4, 6.0 + d)
        img, samples = np.zeros((h, w, 3)), C.c_uint32()
        st = lib.vt_accum_readback(ctx[d], scene, img.ctypes.data, img.size, C.byref(samples))
        assert st == 0, lib.vt_last_error(ctx[d])
        assert samples.value == 4 and np.all(img == (6.0 + d) / 4)
