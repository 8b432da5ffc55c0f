"""The bounded wait of the Newton solve's barrier, run out without a fault: the
blocks of a solve of no points wait for one that does not exist and give up
after a set number of polls.  The call reports IZEM_ERR_TIMEOUT in well under a
second, the state is untouched, and the next solve on the context, whose shared
counters start from zero again, is the oracle's (the bound of
test_gpu_newton_sizes.py)."""
import time

import numpy as np
import pytest

import workloads as W
from phd_gb300 import capi
from phd_gb300.izem import IzemError, IzemGPU

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("polls", [1, 4096, 1 << 16])
def test_newton_barrier_gives_up(polls):
    cfg, thd, adi, dxi, st, info, orc = W.case("mix", 12)
    W.perturb(st, 0.02, seed=5)
    g = IzemGPU(cfg, thd, adi)
    g.set_grid(*dxi)
    g.upload(**st)
    before = g.download()
    for _ in range(2):
        t = time.perf_counter()
        with pytest.raises(IzemError) as e:
            g.newton_wait_selftest(polls)
        assert e.value.code == capi.ERR_TIMEOUT and time.perf_counter() - t < 1.0
    after = g.download()
    for k in ("v", "T", "cp", "ha"):
        np.testing.assert_array_equal(after[k], before[k])
    orc.update_primitives(st)
    g.update_primitives()
    got = g.download()
    it_max, unconverged = g.newton_stats()
    g.close()
    assert it_max > 0 and unconverged == 0
    i = (slice(3, -3),) * 3
    assert np.max(np.abs(got["T"][i] - st["T"][i])) <= 1e-12 * np.max(st["T"])


def test_poll_limits_out_of_range_are_refused():
    cfg, thd, adi, dxi, st, info, orc = W.case("mix", 12)
    g = IzemGPU(cfg, thd, adi)
    for polls in (0, -1, (1 << 20) + 1):
        with pytest.raises(IzemError) as e:
            g.newton_wait_selftest(polls)
        assert e.value.code == capi.ERR_ARG
    g.close()
