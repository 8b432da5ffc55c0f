"""Batches of reactors around the sizes where the launch of the persistent
integrator changes: part of a warp, several one-warp blocks, the full grid's
threads (seven blocks of 128 an SM) less and more one.

A reactor's integration depends on nothing but its own state, so the first n
reactors of a large batch have the results of a batch of n: the same bits."""
import numpy as np
import pytest
import torch

from phd_gb300 import ics
from phd_gb300.izem import psr_batch
from phd_gb300.mech import h2_mechanism

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def large():
    mech = h2_mechanism()
    start = ics.batched_reactors(1 << 18, seed=17)
    T, rho, Y, dt = (a.copy() for a in start)
    istate, nsteps, _ = psr_batch(mech, T, rho, Y, dt)
    return mech, start, T, Y, istate, nsteps


@pytest.mark.parametrize("n", [1, 31, 33, 4097, "full-1", "full", "full+1"])
def test_batch_sizes(large, n):
    mech, start, T1, Y1, is1, ns1 = large
    if isinstance(n, str):
        full = 7 * 128 * torch.cuda.get_device_properties(0).multi_processor_count
        n = full + {"full-1": -1, "full": 0, "full+1": 1}[n]
    T, rho, Y, dt = (a[:n].copy() for a in start)
    istate, nsteps, _ = psr_batch(mech, T, rho, Y, dt)
    np.testing.assert_array_equal(istate, is1[:n])
    np.testing.assert_array_equal(nsteps, ns1[:n])
    np.testing.assert_array_equal(T, T1[:n])
    np.testing.assert_array_equal(Y, Y1[:n])
