"""fmath.cuh against 80-bit or wider host arithmetic.

Bounds.  exp: the fixed-point argument is off by 2^-56 at most for |x| < 128
(2^-59 for |x| < 16), i.e. 2^-56 ln 2 of the result or 0.09 ulp of its lower
end (0.02), on top of the 0.5 ulp of the rounding and 2^-60 of the polynomial
and the table products: 0.62 ulp, 0.53 ulp for |x| < 16.  log: 2^-60 absolute
and the rounding: 0.52 ulp where |log x| >= 1/2.  x^y: 2^-59 of the exponent
and the rounding: 0.55 ulp.  1/x: the seed's 2^-19.4 cubed, two roundings of
small terms and the last one: 0.6 ulp; a/x: 0.51 ulp."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
SRC = os.path.join(HERE, "harness", "fmath_harness.cu")
EXP, LOG, ROOT, RCP, DIV = range(5)


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    nvcc = "/usr/local/cuda/bin/nvcc" if os.path.exists("/usr/local/cuda/bin/nvcc") else "nvcc"
    so = str(tmp_path_factory.mktemp("fmath") / "libfmath.so")
    subprocess.check_call([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O2", "-std=c++17", "-Xcompiler",
                           "-fPIC", "-shared", SRC, "-o", so])
    return C.CDLL(so)


def apply(fn, op, a, b=None):
    a = np.ascontiguousarray(a, dtype=np.float64)
    b = np.ones_like(a) if b is None else np.ascontiguousarray(b, dtype=np.float64)
    y = np.zeros_like(a)
    p = C.POINTER(C.c_double)
    rc = fn(C.c_int(op), C.c_longlong(len(a)), a.ctypes.data_as(p), b.ctypes.data_as(p), y.ctypes.data_as(p))
    assert rc == 0
    return y


def ulps(got, ref):
    ref64 = ref.astype(np.float64)
    return np.abs((got.astype(np.longdouble) - ref) / np.spacing(np.abs(ref64))).max()


def arguments(op):
    """Random arguments over the range in use, with the ends of the tables'
    intervals and of the fixed-point range among them."""
    rng = np.random.Generator(np.random.PCG64(11))
    n = 200000
    if op == EXP:
        x = np.concatenate([rng.uniform(-127.9, 127.9, n), rng.uniform(-16, 16, n), rng.standard_normal(n) * 1e-9,
                            np.arange(-3000, 3000) * (np.log(2.0) / 128.0)])
        x = np.concatenate([x, np.nextafter(x[-6000:], 1e9), np.nextafter(x[-6000:], -1e9),
                            [0.0, -0.0, 1e-300, -1e-300, 5e-324, 127.99999999999999, -127.99999999999999]])
        return x, None
    if op == LOG:
        x = np.concatenate([10.0 ** rng.uniform(-300, 300, n), rng.uniform(200.0, 4000.0, n)])
        k = np.repeat(1.0 + np.arange(128) / 128.0, 3) * np.tile([1.0, 2.0, 1024.0], 128)
        x = np.concatenate([x, k, np.nextafter(k, 0.0), np.nextafter(k, 1e9)])
        return x[np.abs(np.log(x)) >= 0.5], None
    if op == ROOT:
        x = 10.0 ** rng.uniform(-30, 12, n)
        return x, 1.0 / rng.integers(1, 8, n)
    x = np.concatenate([10.0 ** rng.uniform(-120, 120, n), rng.uniform(1.0, 2.0, n)]) * rng.choice([-1.0, 1.0], 2 * n)
    return x, 10.0 ** rng.uniform(-25, 25, 2 * n)


def exact(op, a, b):
    a = a.astype(np.longdouble)
    if op == EXP:
        return np.exp(a)
    if op == LOG:
        return np.log(a)
    if op == ROOT:
        return a ** (b.astype(np.longdouble))
    return 1 / a if op == RCP else a / b.astype(np.longdouble)


BOUND = {EXP: 0.62, LOG: 0.52, ROOT: 0.55, RCP: 0.6, DIV: 0.51}


def check(fn, op):
    a, b = arguments(op)
    got = apply(fn, op, a, b)
    assert ulps(got, exact(op, a, b)) <= BOUND[op]
    if op == EXP:
        s = np.abs(a) < 16
        assert ulps(got[s], exact(op, a[s], b)) <= 0.53


def check_limits(fn):
    inf, nan = np.inf, np.nan
    x = np.array([0.0, -0.0, -800.0, -inf, inf, 710.0, nan, 700.0, -740.0])
    assert np.array_equal(apply(fn, EXP, x)[:6], [1.0, 1.0, 0.0, 0.0, inf, inf])
    assert np.isnan(apply(fn, EXP, x)[6])
    assert np.allclose(apply(fn, EXP, x)[7:], np.exp(x[7:]), rtol=1e-14, atol=1e-323)
    x = np.array([1.0, 0.0, -1.0, inf, nan, 5e-324])
    y = apply(fn, LOG, x)
    assert y[0] == 0.0 and y[1] == -inf and np.isnan(y[2]) and y[3] == inf and np.isnan(y[4])
    assert abs(y[5] / np.log(5e-324) - 1) < 1e-15
    y = apply(fn, ROOT, [0.0, 1.0, inf, 2.0, 4.0], [0.5, 0.3, 0.5, 1.0, 0.5])
    assert np.array_equal(y, [0.0, 1.0, inf, 2.0, 2.0])


@pytest.mark.parametrize("op", [EXP, LOG, ROOT])
def test_host(lib, op):
    if np.finfo(np.longdouble).nmant < 63:
        pytest.skip("no wider host type")
    check(lib.fmath_host, op)
    check_limits(lib.fmath_host)


@pytest.mark.gpu
@pytest.mark.parametrize("op", [EXP, LOG, ROOT, RCP, DIV])
def test_device(lib, op):
    check(lib.fmath_device, op)
    check_limits(lib.fmath_device)
    if op in (RCP, DIV):   # outside the seed's range: the library's value
        a = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, 1e308, -1e300, 1e-290])
        with np.errstate(all="ignore"):
            got, ref = apply(lib.fmath_device, RCP, a), 1.0 / a
            assert np.array_equal(got, ref, equal_nan=True)
            got, ref = apply(lib.fmath_device, DIV, a, a[::-1]), a / a[::-1]
            assert np.array_equal(got, ref, equal_nan=True)
    else:   # the device computes the host compilation's bits
        a, b = arguments(op)
        assert np.array_equal(apply(lib.fmath_device, op, a, b), apply(lib.fmath_host, op, a, b))
