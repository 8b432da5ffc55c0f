"""Two contexts of one species set stepped by two threads at once: each Newton
solve is a cooperative launch on its context's own stream, with its own shared
state (the larger block's launches fill the GPU), so the results are those of
the contexts stepped one after the other, to the bit."""
import threading

import numpy as np
import pytest

import workloads as W
from phd_gb300.izem import IzemGPU

pytestmark = pytest.mark.gpu


def _context(name, n):
    cfg, thd, adi, dxi, st, info, orc = W.case(name, n)
    g = IzemGPU(cfg, thd, adi)
    g.set_grid(*dxi)
    g.upload(**st)
    return g


def _steps(g, n):
    for _ in range(n):
        g.rk3(g.timestep()[1])


@pytest.mark.parametrize("small,large,steps", [(("mix", 16), ("mix", 64), 12)])
def test_two_contexts_at_once(small, large, steps):
    want = []
    for name, n in (small, large):
        g = _context(name, n)
        _steps(g, steps)
        want.append(g.download())
        g.close()
    gs = [_context(*small), _context(*large)]
    errors = []

    def run(g):
        try:
            _steps(g, steps)
        except Exception as e:   # reported in the main thread
            errors.append(e)

    threads = [threading.Thread(target=run, args=(g,)) for g in gs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for g, w in zip(gs, want):
        got = g.download()
        g.close()
        for k in ("v", "T"):
            np.testing.assert_array_equal(got[k], w[k])
