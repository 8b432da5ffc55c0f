"""The mole fractions of the point kernels, X = (rho Y / W) / (rho W_i) with one
shared reciprocal, against wider host arithmetic.

Bound: one rounding of a value spread evenly over a binade's logarithm has an
rms of sqrt(3 / (8 ln 2) / 3) = 0.425 units of 2^-53.  X takes two (the product
with 1 / W, the last one), 0.60; the quotient (rho Y) / (rho W_i W) takes three,
0.74, and must not be more accurate."""
import ctypes as C
import os
import re
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "phd_gb300", "csrc")


@pytest.mark.gpu
def test_rounding_of_the_shared_reciprocal(tmp_path):
    nvcc = "/usr/local/cuda/bin/nvcc" if os.path.exists("/usr/local/cuda/bin/nvcc") else "nvcc"
    so = str(tmp_path / "libmolefrac.so")
    subprocess.check_call([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O2", "-std=c++17", "-Xcompiler",
                           "-fPIC", "-shared", os.path.join(HERE, "harness", "molefrac_harness.cu"), "-o", so])
    rng = np.random.Generator(np.random.PCG64(5))
    n = 200000
    rho, Wi = 10.0 ** rng.uniform(-2, 1, n), 10.0 ** rng.uniform(-1, 1, n)
    rY, W_i = rho * 10.0 ** rng.uniform(-12, 0, n), 10.0 ** rng.uniform(-1, 1, n)
    a, y = rY * W_i, np.zeros(n)
    p = C.POINTER(C.c_double)
    rc = C.CDLL(so).molefrac_device(C.c_int(n), *(q.ctypes.data_as(p) for q in (a, rho, Wi, y)))
    assert rc == 0
    wide = np.longdouble
    ref = rY.astype(wide) * W_i.astype(wide) / (rho.astype(wide) * Wi.astype(wide))
    rms = float(np.sqrt(np.mean(((y.astype(wide) - ref) / ref) ** 2))) * 2.0 ** 53
    assert rms <= 0.65, rms


def test_the_fourier_criteria_take_the_same_mole_fractions():
    """k_dtv and k_prim form X_k by the same function."""
    for name, kernel in (("kernels_state.cuh", "k_dtv"), ("kernels_euler.cuh", "k_prim")):
        body = open(os.path.join(CSRC, name)).read().split("void %s(" % kernel)[1].split("__global__")[0]
        assert "fm_rcp_prod(rho, Wi)" in body and len(re.findall(r"\bfm_over\(v\[|\bfm_over\(rY", body)) == 1, kernel
