"""A fetch of many pixels goes through a bounded device buffer, and its pieces are the oracle's pixels."""

import numpy as np
import pytest

from opengate_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def test_large_projections_take_little_device_memory(built_lib):
    import torch

    from opengate_gb300.engine import SpectEngine
    from oracle import oracle as O

    scene, sp, _ = W.spect_phantom(shape=(20, 32, 32), spacing=9.6, n_runs=18)
    sp.size, sp.spacing = [511, 512], [565.76 / 511, 565.76 / 512]
    sp.set_free_flight()
    n = int(np.prod(sp.projection_shape()))
    assert 8 * n > 140e6  # more than the buffer may take, and not a whole number of its pieces
    with SpectEngine(scene, sp) as eng:
        eng.run(1000, 11)
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        w, w2 = eng.weighted_projection(squared=True)
        taken = free - torch.cuda.mem_get_info()[0]
        counters = eng.counters()
    assert taken <= 144e6, taken  # 128 MiB, and what loading the kernel may take
    rw, rw2, rcnt = O.run_spect_ff(scene, sp, 1000, seed=11, threads=8)
    assert counters == rcnt and rw.any()
    assert np.array_equal(w, rw) and np.array_equal(w2, rw2)
