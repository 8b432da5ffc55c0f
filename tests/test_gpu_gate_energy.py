"""The gated surrogate step's energy-consistent temperature on both sides of
and across the middle temperature of the thermodynamic fits (1000 K), against
64-bit host arithmetic.

The network is zero, so that its prediction is the output mean: a conversion
of hydrogen to water and a temperature increment that is off by 3 K.  The gate
takes every cell (its tolerances are wide); the accepted temperature solves
e(T1, Y1) = e(T0, Y0).  Bound: four Newton steps from 3 K away leave less than
1e-14 of T; e sums nine terms of up to 1e11 erg/g with roundings of 2^-53
each, over c_v of 1e7: 1e-9 K at most.  The fits of the two ranges differ by
up to 1e-5 of c_v T at 1000 K, so no cell may end within 0.1 K of it."""
import numpy as np
import pytest

from phd_gb300 import ics
from phd_gb300.mech import h2_mechanism
from phd_gb300.surrogate import Surrogate
from phd_gb300.thd import load_species

pytestmark = pytest.mark.gpu


def _energy(m, T, Y):
    e = np.zeros_like(T)
    for k in range(m.kk):
        a = np.where((T > m.tmid[k])[:, None], np.array(list(m.a[k][1])), np.array(list(m.a[k][0])))
        h = a[:, 5] + T * (a[:, 0] + T * (a[:, 1] / 2 + T * (a[:, 2] / 3 + T * (a[:, 3] / 4 + T * a[:, 4] / 5))))
        e += Y[:, k] * m.ru / m.wt[k] * (h - T)
    return e


# 828: the iterations start above 1000 K, some of them end below
@pytest.mark.parametrize("T0", [700.0, 828.0, 850.0, 1100.0])
def test_accepted_temperature(T0):
    m = h2_mechanism()
    n = 1000
    _, rho, Y, dt = ics.batched_reactors(n, seed=11)
    T = T0 + np.linspace(0.0, 3.0, n)
    names = ["H2", "O2", "H2O"]
    idx = [load_species("h2air9")["names"].index(s) for s in names]
    ox = 0.05
    Y[:] = 0.0
    Y[:, idx[0]], Y[:, idx[1]], Y[:, idx[2]] = 0.05, 0.25, 0.1
    Y[:, -1] = 0.6
    dY = np.zeros(10)
    w = np.array([m.wt[k] for k in range(m.kk)])
    for k, nu in zip(idx, (-2.0, -1.0, 2.0)):
        dY[k] = nu * w[k] * ox * 0.01
    # the increment by a converged host solution for the middle cell, 3 K off
    Y1 = Y + dY[:9]
    Y1 /= Y1.sum(axis=1, keepdims=True)
    e0 = _energy(m, T, Y)
    ref = T + 20.0
    for _ in range(60):
        ref = ref - (_energy(m, ref, Y1) - e0) / ((_energy(m, ref + 0.01, Y1) - _energy(m, ref - 0.01, Y1)) / 0.02)
    keep = np.abs(ref - 1000.0) > 0.1
    norm = np.zeros(44, dtype=np.float32)
    norm[12:24] = 1.0
    norm[34:44] = 1.0
    norm[24:33] = dY[:9]
    norm[33] = float(np.median(ref - T) + 3.0)
    s = Surrogate(seed=1)
    W, b = s.get_params()
    s.set_params([np.zeros_like(a) for a in W], [np.zeros_like(a) for a in b])
    s.set_norm(norm)
    gate = (300.0, 3000.0, 0.0, 1.0, 1.0, 1e3, 1.0, 1e3, 1.0, 1e3)
    # what the device adds is the FP32 mean
    Y1 = Y + norm[24:33].astype(np.float64)
    Y1 /= Y1.sum(axis=1, keepdims=True)
    for _ in range(60):
        ref = ref - (_energy(m, ref, Y1) - e0) / ((_energy(m, ref + 0.01, Y1) - _energy(m, ref - 0.01, Y1)) / 0.02)
    T1, Yn = T.copy(), Y.copy()
    r = s.chem_step(m, T1, rho.copy(), Yn, dt.copy(), gate)
    assert r["fallback"] == 0
    assert np.abs(Yn - Y1).max() <= 1e-15
    assert (ref > T).all() and keep.sum() > n // 2
    assert np.abs(T1 - ref)[keep].max() <= 1e-9
