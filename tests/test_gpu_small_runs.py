"""Runs of a few histories: the pooled transport against the compacted wavefront's.

Their launch is the set-up of a block and the longest history; both kernels run the same events, so
neither may take much longer.  The wavefront kernel's block has 256 threads whatever the run.
"""

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
