"""The FFT passes of the kernels (phaser_b200/csrc/fft_pass.cuh) alone against numpy, forward and inverse, through a
test-only library (tests/cuda/pass_selftest.cu) linked against the product library: compile-time plans; runtime plans in
every radix order (prime radices first, last and alone), from global and from shared memory, one and two sequences an
item; a last block with unused columns.  Bar: that of the shared-memory engines (FP32 transform error)."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def lib():
    from phaser_b200 import build
    prod = build.build()
    src, out = os.path.join(HERE, "cuda", "pass_selftest.cu"), os.path.join(HERE, "_build")
    os.makedirs(out, exist_ok=True)
    so = os.path.join(out, "libphaser_pass_selftest.so")
    deps = [src, prod] + [os.path.join(build.CSRC, f) for f in os.listdir(build.CSRC) if f.endswith((".cuh", ".h"))]
    if not os.path.exists(so) or any(os.path.getmtime(d) > os.path.getmtime(so) for d in deps):
        libdir = os.path.dirname(prod)
        subprocess.run([build.nvcc()] + build.ARCH + build.NVCC_FLAGS +
                       ["-shared", src, "-o", so, "-L" + libdir, "-lphaser_gpu", "-Xlinker", "-rpath=" + libdir],
                       check=True, capture_output=True, text=True)
    lib = C.CDLL(so)
    lib.phgpu_selftest_pass.argtypes = [C.c_int] * 5 + [C.c_void_p]
    return lib


def check(lib, n, inverse, mode, order=0):
    rng = np.random.default_rng(n)
    x = (rng.standard_normal((7, n)) + 1j * rng.standard_normal((7, n))).astype(np.complex64)
    y = x.copy()
    assert lib.phgpu_selftest_pass(n, len(x), inverse, mode, order, y.ctypes.data) == 0
    ref = np.fft.ifft(x.astype(np.complex128), axis=1) * n if inverse else np.fft.fft(x.astype(np.complex128), axis=1)
    err = np.abs(y - ref).max() / np.abs(ref).max()
    assert err < 5e-6, (n, inverse, mode, order, err)


@pytest.mark.parametrize("n", [64, 128, 200, 256, 320, 512])
@pytest.mark.parametrize("inverse", [0, 1])
def test_compile_time_plans(lib, n, inverse):
    check(lib, n, inverse, 0)


@pytest.mark.parametrize("n", [1, 2, 3, 8, 11, 13, 30, 64, 77, 97, 100, 121, 127, 134, 143, 169, 201, 242, 254, 286, 360, 381, 512,
                               889, 1016, 1024])
@pytest.mark.parametrize("mode", [1, 2, 3])
def test_runtime_plans(lib, n, mode):
    for order in range(3):
        for inverse in (0, 1):
            check(lib, n, inverse, mode, order)
