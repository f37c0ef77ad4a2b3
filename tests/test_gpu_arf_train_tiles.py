"""Training steps at the edges of their tiles: one tile, a whole wave of SMs, more than one wave.

A step is exact up to the storage points it shares with the oracle: the gradient of a batch is
compared with the FP64 oracle's (BF16 rounding emulated), and the order in which tiles and kernels
overlap changes nothing (two trainings of the same rows give the same weights).
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _engine():
    from opengate_gb300 import workloads as W
    from opengate_gb300.engine import SpectEngine

    scene, sp, _ = W.spect_phantom(shape=(4, 8, 8), spacing=40.0, n_runs=1)
    return SpectEngine(scene, sp)


def _rows(n, seed=3):
    rng = np.random.default_rng(seed)
    r = np.empty((n, 4), np.float32)
    r[:, 0] = rng.uniform(0.1, 0.16, n)
    r[:, 1] = rng.uniform(0.0, 60.0, n)
    r[:, 2] = rng.uniform(-180.0, 180.0, n)
    r[:, 3] = rng.integers(0, 3, n)
    return r


@pytest.mark.parametrize("batch,n", [(128, 130), (128 * 8, 5000), (128 * 133, 20_000), (128 * 152, 40_001),
                                     (128 * 200, 30_000)])
def test_training_is_reproducible_and_learns(built_lib, batch, n):
    from opengate_gb300.engine import ArfNetwork

    rows = _rows(n)
    rows[:, 3] = (rows[:, 1] > 30.0) + (rows[:, 0] > 0.13)  # a class the inputs decide
    out = []
    for _ in range(2):
        with _engine() as eng:
            net = ArfNetwork(eng)
            _, loss = net.train_rows(rows, 0.1, 0.16, 60.0, 2.0, epochs=6, batch=batch, lr=3e-3)
            out.append((net.params(), loss))
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
    assert np.isfinite(out[0][0]).all() and loss[-1] < loss[0]


@pytest.mark.parametrize("bad,at", [(np.nan, 0), (np.inf, 2), (3.0, 3), (-1.0, 3), (0.5, 3)])
def test_bad_rows_are_named(built_lib, bad, at):
    from opengate_gb300.engine import ArfNetwork

    rows = _rows(700)
    rows[611, at] = rows[690, at] = bad
    with _engine() as eng, pytest.raises(Exception, match="row 611"):
        ArfNetwork(eng).train_rows(rows, 0.1, 0.16, 60.0, 2.0, epochs=1, batch=128)
