"""fm_log between e^-1/2 and e^1/2, its relative error there.

The fixed-point logarithm has an absolute error below 2^-61, which would be any
number of units of the last place near 1, where log x itself vanishes.  Bounds:
for |x - 1| >= 2^-6 the result is at least 2^-7, whose last place is 2^-59: half
of it for the rounding and 2^-61 / 2^-59, 0.75.  Nearer to 1 the library's
logarithm: 1 (CUDA's bound; the host's is below)."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
LOG = 1


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    nvcc = "/usr/local/cuda/bin/nvcc" if os.path.exists("/usr/local/cuda/bin/nvcc") else "nvcc"
    so = str(tmp_path_factory.mktemp("fmath") / "libfmath.so")
    subprocess.check_call([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O2", "-std=c++17", "-Xcompiler",
                           "-fPIC", "-shared", os.path.join(HERE, "harness", "fmath_harness.cu"), "-o", so])
    return C.CDLL(so)


def arguments():
    rng = np.random.Generator(np.random.PCG64(23))
    n = 100000
    d = 10.0 ** rng.uniform(-16, -0.5, n)
    ends = np.concatenate([1.0 + 2.0 ** -np.arange(2, 53), 1.0 - 2.0 ** -np.arange(2, 54)])
    x = np.concatenate([1.0 + d, 1.0 - d, rng.uniform(1 - 2.0 ** -5, 1 + 2.0 ** -5, n), rng.uniform(0.61, 1.64, n),
                        ends, np.nextafter(ends, 0.0), np.nextafter(ends, 2.0)])
    return x[(x != 1.0) & (np.abs(np.log(x)) < 0.5)]


def check(fn):
    x = np.ascontiguousarray(arguments())
    y = np.zeros_like(x)
    p = C.POINTER(C.c_double)
    assert fn(C.c_int(LOG), C.c_longlong(len(x)), x.ctypes.data_as(p), x.ctypes.data_as(p), y.ctypes.data_as(p)) == 0
    ref = np.log(x.astype(np.longdouble))
    err = np.abs((y.astype(np.longdouble) - ref) / np.spacing(np.abs(ref.astype(np.float64))))
    near = np.abs(x - 1.0) < 2.0 ** -6
    assert err[near].max() <= 1.0, (x[near][err[near].argmax()], err[near].max())
    assert err[~near].max() <= 0.75, (x[~near][err[~near].argmax()], err[~near].max())


def test_host(lib):
    if np.finfo(np.longdouble).nmant < 63:
        pytest.skip("no wider host type")
    check(lib.fmath_host)


@pytest.mark.gpu
def test_device(lib):
    check(lib.fmath_device)
