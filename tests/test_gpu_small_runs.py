"""Runs of a few histories: the pooled transport against the compacted wavefront's.

Their launch is the set-up of a block and the longest history; both kernels run the same events, so
neither may take much longer.  The wavefront kernel's block has 256 threads whatever the run.
"""

import numpy as np
import pytest

from opengate_gb300 import _capi as C
from opengate_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def _transport_ms(scene, kernel, n, **opts):
    from opengate_gb300.engine import DoseEngine

    with DoseEngine(scene, **opts) as eng:
        eng.set_transport_kernel(kernel)
        best = float("inf")
        for _ in range(20):
            eng.reset()
            eng.run(n, 5)
            best = min(best, eng.last_kernel_ms()[1])
    return best


def test_one_history_does_not_wait_for_the_tables(built_lib):
    """57 KB of tables copied by the run's one warp: 51 us with one load at a time (wavefront 29), 25 with eight."""
    scene, _ = W.ct_phantom(shape=(80, 128, 128), spacing=2.4)
    pooled, wavefront = (_transport_ms(scene, k, 1) for k in (C.GG_KERNEL_PHASED, C.GG_KERNEL_WAVEFRONT))
    assert pooled < 1.3 * wavefront, (pooled, wavefront)


def test_a_warp_of_histories_is_spread_over_the_gangs(built_lib):
    """32 FP64 histories: 391 us in one gang (wavefront 270); no gang holds more than one when they are spread."""
    scene, _ = W.ct_phantom(shape=(80, 128, 128), spacing=2.4)
    pooled, wavefront = (_transport_ms(scene, k, 32, precision=64) for k in (C.GG_KERNEL_PHASED, C.GG_KERNEL_WAVEFRONT))
    assert pooled < 1.2 * wavefront, (pooled, wavefront)


@pytest.mark.parametrize("n", [2, 10, 151, 153, 1000, 4863])
def test_few_histories_bit_exact(built_lib, n):
    from opengate_gb300.engine import DoseEngine
    from oracle import oracle as O

    scene, _ = W.ct_phantom(shape=(40, 64, 64), spacing=4.8)
    with DoseEngine(scene) as eng:
        eng.run(n, 19, 3)
        got = eng.edep(), eng.edep_squared(), eng.counters()
    ref = O.run_dose(scene, n, 19, first=3, threads=4)
    assert got[2] == ref[2]
    assert np.array_equal(got[0], ref[0]) and np.array_equal(got[1], ref[1])
