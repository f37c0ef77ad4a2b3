"""Launch options of a dose run: they bound nothing that the pooled kernel needs for its speed.

The option block_size is the head stage's; a run with small blocks takes the transport as long as
one with the default (it took 2 to 9 times as long when the option capped the threads of an SM).
"""

import pytest

from opengate_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def _transport_ms(scene, **opts):
    from opengate_gb300.engine import DoseEngine

    with DoseEngine(scene, **opts) as eng:
        best = float("inf")
        for _ in range(4):
            eng.reset()
            eng.run(10_000_000, 3)
            best = min(best, eng.last_kernel_ms()[1])
    return best


@pytest.mark.parametrize("block_size,blocks_per_sm", [(32, 0), (64, 0), (128, 0), (128, 1), (256, 0)])
def test_small_blocks_do_not_slow_the_transport(built_lib, block_size, blocks_per_sm):
    scene, _ = W.ct_phantom(shape=(80, 128, 128), spacing=2.4)
    ref = _transport_ms(scene)
    got = _transport_ms(scene, block_size=block_size, blocks_per_sm=blocks_per_sm)
    assert got < 1.5 * ref, (got, ref)
