"""Nothing of a network handle is shared by handles of other devices or threads.

A kernel's shared-memory limit belongs to a device, so a process-wide flag for
"already raised" would leave it at the default for the handles of a second
device, whose launches then fail.  One GPU cannot show that: the first test
reads the sources."""
import glob
import os
import re
import threading

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "phd_gb300", "csrc")


def test_no_process_wide_flags():
    for path in glob.glob(os.path.join(CSRC, "*.cu*")):
        text = open(path).read()
        assert re.findall(r"\bstatic\s+(?:bool|std::once_flag|std::atomic\S*)\s+\w+\s*[;={]", text) == [], path


def _train(seed):
    from phd_gb300.surrogate import Surrogate
    s = Surrogate(seed=seed)
    rng = np.random.Generator(np.random.PCG64(seed))
    x, t = rng.standard_normal((2048, 12)).astype(np.float32), rng.standard_normal((2048, 10)).astype(np.float32)
    s.train(x, t, epochs=2, batch=512)
    p = s.get_params()
    s.close()
    return p


@pytest.mark.gpu
def test_two_handles_trained_at_once():
    """Weights after training in two threads are those of one after the other, to the bit."""
    want = [_train(31), _train(32)]
    got, errors = [None, None], []

    def run(q):
        try:
            got[q] = _train(31 + q)
        except Exception as e:   # reported in the main thread
            errors.append(e)

    threads = [threading.Thread(target=run, args=(q,)) for q in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for w, g in zip(want, got):
        for a, b in zip(w[0] + w[1], g[0] + g[1]):
            np.testing.assert_array_equal(a, b)
