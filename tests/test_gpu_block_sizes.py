"""A time step of grids on both sides of the sizes where the point kernels
change their threads per block (8 and 32 warps an SM), against the oracle.

The state and the bounds are those of the other RK3 tests: 2 % noise on the
conserved variables, so that no component of the update is a difference of
equal fluxes, and 1e-12 of a variable's largest value.  The time step is a
maximum over points of some twenty rounded operations, two square roots and a
quotient among them: 1e-14."""
import numpy as np
import pytest
import torch

import workloads as W
from phd_gb300.izem import IzemGPU

pytestmark = pytest.mark.gpu


# points n^3 just below (-) and at or above (+) the line
@pytest.mark.parametrize("warps,side", [(8, "-"), (8, "+"), (32, "-"), (32, "+")])
def test_step_around_the_block_size_lines(warps, side):
    line = warps * 32 * torch.cuda.get_device_properties(0).multi_processor_count
    n = int(np.ceil(line ** (1.0 / 3.0))) - (side == "-")
    cfg, thd, adi, dxi, st, info, orc = W.case("tgv", n)
    W.perturb(st, 0.02, seed=3)
    orc.update_primitives(st)
    g = IzemGPU(cfg, thd, adi)
    g.set_grid(*dxi)
    g.upload(**st)
    _, dt = orc.timestep(st)
    _, dtg = g.timestep()
    orc.rk3(st, dt)
    g.rk3(dt)
    got = g.download()
    g.close()
    assert abs(dtg - dt) <= 1e-14 * abs(dt)
    i = (slice(3, -3),) * 3
    err = W.normwise(got["v"][i], st["v"][i])
    assert np.all(err <= 1e-12), err
