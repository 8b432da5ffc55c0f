"""Loss and parameter gradients of the surrogate at batch sizes around the
tiles and splits of the training GEMMs (128 rows a tile, 64 a K chunk, at
most 32 splits of the batch), and two Adam steps on them.

Tolerances as in test_gpu_mlp.py: operands are BF16 on both sides, which
leaves 3e-2 of a gradient's norm; the Adam steps are then taken from the
device's own gradients in FP64, where each FP32 step rounds a weight by half
a unit in the last place and its increment, at most 2 lr in magnitude, by a
few (16 x 2^-24) and by what 1 - 0.999^step loses as an FP32 difference (6e-5)."""
import numpy as np
import pytest

from oracle import mlp_oracle as mo
from phd_gb300.surrogate import Surrogate

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 63, 128, 129, 1000, 2176, 4097])
def test_gradients_and_adam_steps(M):
    rng = np.random.Generator(np.random.PCG64(M))
    x = rng.standard_normal((M, 12)).astype(np.float32)
    t = rng.standard_normal((M, 10)).astype(np.float32)
    s = Surrogate(seed=21)
    lr, b1, b2, eps = 1e-3, np.float32(0.9), np.float32(0.999), 1e-8
    P = [np.asarray(a, np.float64) for side in s.get_params() for a in side]
    m = [np.zeros_like(p) for p in P]
    v = [np.zeros_like(p) for p in P]
    for step in (1, 2):
        W, b = s.get_params()
        loss, gW, gb = s.grads(x, t)
        lref, rW, rb = mo.loss_and_grads(W, b, x, t)
        assert abs(loss - lref) <= 1e-2 * lref
        for g, r in zip(list(gW) + list(gb), list(rW) + list(rb)):
            assert np.linalg.norm(g - r) <= 3e-2 * np.linalg.norm(r)
        P = [np.asarray(a, np.float64) for a in list(W) + list(b)]
        losses = s.train(x, t, epochs=1, batch=M, lr=lr)
        assert abs(losses[0] - loss) <= 1e-12 * loss
        c1, c2 = 1.0 - float(b1) ** step, 1.0 - float(b2) ** step
        for k, (g, new) in enumerate(zip(list(gW) + list(gb), [a for side in s.get_params() for a in side])):
            g = np.asarray(g, np.float64)
            m[k] = float(b1) * m[k] + (1.0 - float(b1)) * g
            v[k] = float(b2) * v[k] + (1.0 - float(b2)) * g * g
            ref = P[k] - lr * (m[k] / c1) / (np.sqrt(v[k] / c2) + eps)
            assert np.all(np.abs(new - ref) <= 2.0 ** -23 * np.abs(ref) + (16 * 2.0 ** -24 + 6e-5) * 2.0 * lr)


# rows around one tile of 128, several tiles and a ragged end, more tiles than SMs
@pytest.mark.parametrize("M", [1, 127, 129, 1000, 152 * 128 + 37])
def test_forward_rows(M):
    rng = np.random.Generator(np.random.PCG64(100 + M))
    x = rng.standard_normal((M, 12)).astype(np.float32)
    s = Surrogate(seed=22)
    W, b = s.get_params()
    b = [rng.standard_normal(a.shape).astype(np.float32) * 0.1 for a in b]
    s.set_params(W, b)
    y = s.forward(x)
    assert y.shape == (M, 10)
    ref, _ = mo.forward(W, b, x)
    # BF16 operands on both sides: 1e-2 of the largest output, as in test_gpu_mlp.py
    assert np.abs(y - ref).max() <= 1e-2 * np.abs(ref).max()
