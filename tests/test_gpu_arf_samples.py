"""ARF training rows at the edges of the sampler's warps and blocks, against the CPU oracle.

Energies and classes are bit-exact.  The angles are not compared here: the device takes them from
the FP32 cosine (in FP64 runs too), the oracle from the cosine it has.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,precision,roulette,first", [
    (1, 32, 1.0, 0), (31, 32, 4.0, 5), (33, 32, 1.0, 0), (256, 32, 1.0, 1 << 33), (257, 64, 3.0, 0),
    (152 * 6 * 256 + 1, 32, 50.0, 3), (2049, 64, 1.0, 0),
])
def test_samples_equal_the_oracles(built_lib, n, precision, roulette, first):
    from opengate_gb300 import workloads as W
    from opengate_gb300.engine import ArfNetwork, SpectEngine
    from oracle import oracle as O

    scene, sp, _ = W.spect_phantom(shape=(4, 8, 8), spacing=40.0, n_runs=1)
    a = ArfNetwork.sampling(0.12, 0.16, 25.0, (150.0, 90.0), roulette)
    with SpectEngine(scene, sp, precision=precision) as eng:
        rows = ArfNetwork(eng).dataset(a, n, seed=21, first=first)
    ref, _ = O.arf_dataset(scene.tables_desc, sp, a, n, seed=21, first=first, threads=4, precision=precision)
    assert np.array_equal(rows[:, [0, 3]], ref[:, [0, 3]])  # energies and classes, in sample order
