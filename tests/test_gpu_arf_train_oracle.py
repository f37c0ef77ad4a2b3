"""Adam steps of the ARF training against the FP64 oracle, at tile counts on both sides of the rule that
overlaps a step's launches (up to 7/8 of a wave of 152 SMs, and the last wave of more).

With eps = 1 Adam's update is lr * m / (1 + sqrt(v)), close to linear in the gradient, so the change of
the weights carries the gradient's own error: the bounds are those of the gradient's test (1 % of the
norm over all, 2 % in a layer, BF16 storage points emulated).
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

M = pytest.importorskip("oracle.arf_mlp")

E_LO, E_HI, THETA = 0.1, 0.16, 60.0
MEAN = (0.5 * THETA, 0.0, 0.5 * (E_LO + E_HI))
STD = (THETA / np.sqrt(12.0), 360.0 / np.sqrt(12.0), (E_HI - E_LO) / np.sqrt(12.0))


def _rows(n):
    rng = np.random.default_rng(n)
    r = np.empty((n, 4), np.float32)
    r[:, 0] = rng.uniform(E_LO, E_HI, n)
    r[:, 1] = rng.uniform(0.0, THETA, n)
    r[:, 2] = rng.uniform(-180.0, 180.0, n)
    r[:, 3] = (r[:, 1] > 30.0).astype(int) + (r[:, 0] > 0.13)
    return r


def _adam(p, rows, batch, epochs, lr, b1=0.9, b2=0.999, eps=1.0):
    n, steps = len(rows), -(-len(rows) // batch)
    m, v, t, losses = np.zeros_like(p), np.zeros_like(p), 0, []
    for _ in range(epochs):
        total = 0.0
        for _ in range(steps):
            at = (np.arange(batch) + t * batch % n) % n
            loss, g = M.loss_and_grad(p, rows[at], MEAN, STD, 3, bf16_points=True)
            t += 1
            m, v = b1 * m + (1 - b1) * g, b2 * v + (1 - b2) * g * g
            p = p - lr * (m / (1 - b1 ** t)) / (np.sqrt(v / (1 - b2 ** t)) + eps)
            total += loss
        losses.append(total / steps)
    return p, losses


@pytest.mark.parametrize("tiles,rows,epochs", [(1, 300, 2), (8, 3000, 1), (133, 30_000, 1), (134, 30_000, 1),
                                               (152, 25_000, 1), (200, 30_000, 2)])
def test_weights_after_a_few_steps(built_lib, tiles, rows, epochs):
    from opengate_gb300 import workloads as W
    from opengate_gb300.engine import ArfNetwork, SpectEngine

    scene, sp, _ = W.spect_phantom(shape=(4, 8, 8), spacing=40.0, n_runs=1)
    data, kw = _rows(rows), dict(batch=128 * tiles, init_seed=5, eps=1.0)
    with SpectEngine(scene, sp) as eng:
        net = ArfNetwork(eng)
        net.train_rows(data, E_LO, E_HI, THETA, 1.0, epochs=1, lr=1e-30, lr_final=1e-30, **kw)
        start = net.params().astype(np.float64)  # (steps of 1e-30 move no FP32 weight)
        _, loss = net.train_rows(data, E_LO, E_HI, THETA, 1.0, epochs=epochs, lr=0.5, lr_final=0.5, **kw)
        change = net.params().astype(np.float64) - start
    ref, ref_loss = _adam(start, data, 128 * tiles, epochs, 0.5)
    ref = ref - start
    np.testing.assert_allclose(loss, ref_loss, rtol=2e-3)

    def rel(a, b):
        return float(np.linalg.norm(a - b) / np.linalg.norm(b))

    assert rel(change, ref) < 1e-2
    for name, (o, size) in M.OFF.items():
        assert rel(change[o:o + size], ref[o:o + size]) < 2e-2, name
