"""The surrogate's training step at the edges of its 32-sample tiles and of one
tile per CTA: gradient and loss of one batch against the FP64 restatement, and a
few Adam steps over minibatches that do not divide the samples against the same
steps in FP64.

Tolerances: an FP32 gradient entry is a sum of n products with relative rounding
near 1e-7, so the gradient's norm agrees to 1e-4 with room; Adam moves each
weight by at most lr = 1e-3 a step whatever the size of its gradient, and only
entries whose gradient is lost in rounding can move differently, so five steps
leave the weights (norm about 20) within 1e-3 of the FP64 ones in norm.
"""
import numpy as np
import pytest

from oracle import mlp_oracle as M
from qd_b200 import systems as S
from qd_b200.surrogate import Surrogate, training_set

pytestmark = pytest.mark.gpu

MASSES = np.array([18.9984, 1.00783, 1.00783]) * S.AMU_ME


@pytest.mark.parametrize("n", [1, 31, 32, 33, 148 * 32, 148 * 32 + 1, 9999])
def test_gradient_of_one_batch(n):
    data = training_set(S.leps_f_h2(), MASSES, n=n, seed=21)
    with Surrogate(seed=5) as sur:
        w, _ = sur.params()
        norm = np.array([0.2, 0.3, 0.05, 0.2, 0.3, 0.1, 0.05, 0.1], dtype=np.float32)
        sur.set_params(w, norm)
        loss, g = sur.loss_and_grad(*data)
    l_ref, g_ref = M.loss_and_grad(w, norm, *data)
    assert abs(loss - l_ref) < 1e-4 * l_ref
    assert np.linalg.norm(g - g_ref) < 1e-4 * np.linalg.norm(g_ref)


@pytest.mark.parametrize("n,batch", [(100, 40), (70, 70), (5000, 4800)])
def test_adam_steps(n, batch):
    data = training_set(S.leps_f_h2(), MASSES, n=n, seed=22)
    lr, lr_end, steps = 1e-3, 1e-4, 5
    with Surrogate(seed=6) as sur:
        w0, _ = sur.params()
        loss = sur.fit(*data, steps=steps, batch=batch, lr=lr, lr_end=lr_end)
        w, norm = sur.params()
    p, m, v = w0.astype(np.float64), 0.0, 0.0
    s0, total, seen, last = 0, 0.0, 0, None
    for t in range(1, steps + 1):
        part = [a[s0:s0 + batch] for a in data]
        l, g = M.loss_and_grad(p, norm, *part)
        m, v = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
        p = p - lr * (m / (1 - 0.9 ** t)) / (np.sqrt(v / (1 - 0.999 ** t)) + 1e-8)
        lr *= (1e-4 / 1e-3) ** (1 / (steps - 1))
        total, seen = total + l * part[0].size, seen + part[0].size
        last = total / seen
        s0 += part[0].size
        if s0 >= n:
            s0, total, seen = 0, 0.0, 0
    assert np.linalg.norm(w - p) < 1e-3
    assert abs(loss - last) < 1e-3 * last


@pytest.mark.parametrize("n", [1, 63, 255, 257, 148 * 64, 148 * 64 + 1, 148 * 128 + 1, 148 * 256, 148 * 256 + 1, 148 * 512 + 1, 200001])
def test_energies_at_the_edges_of_a_round(n):
    # an FP32 output sums 64 products with relative rounding near 1e-7 over four layers
    data = training_set(S.leps_f_h2(), MASSES, n=n, seed=23)
    with Surrogate(seed=7) as sur:
        w, _ = sur.params()
        norm = np.array([0.2, 0.3, 0.05, 0.2, 0.3, 0.1, 0.05, 0.1], dtype=np.float32)
        sur.set_params(w, norm)
        got = sur(*data[:3])
    ref = M.predict(w, norm, *data[:3])
    assert np.abs(got - ref).max() < 1e-5 * np.abs(ref).max() + 1e-7
