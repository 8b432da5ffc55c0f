"""The Newton solve of blocks with one and with two points to a thread of its
launch (nine species: five blocks of 128 threads an SM), and of a few points,
against the oracle.

Bound: the corrections end below 1e-10 of T, squared by the next iteration;
what is left is the rounding of e(T) - e, some thirty operations, over the
slope: the 1e-12 of the largest T of the other state tests."""
import numpy as np
import pytest
import torch

import workloads as W
from phd_gb300.izem import IzemGPU

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("per_thread", ["few", "one", "two"])
def test_newton_solve_sizes(per_thread):
    full = 640 * torch.cuda.get_device_properties(0).multi_processor_count
    n = {"few": 8, "one": int((1.8 * full) ** (1.0 / 3.0)), "two": int((2.6 * full) ** (1.0 / 3.0))}[per_thread]
    cfg, thd, adi, dxi, st, info, orc = W.case("mix", n)
    W.perturb(st, 0.02, seed=5)
    g = IzemGPU(cfg, thd, adi)
    g.set_grid(*dxi)
    g.upload(**st)
    orc.update_primitives(st)
    g.update_primitives()
    got = g.download()
    g.close()
    i = (slice(3, -3),) * 3
    assert np.max(np.abs(got["T"][i] - st["T"][i])) <= 1e-12 * np.max(st["T"])
