"""The pooled transport kernel at the edges of its rounds, against the CPU oracle (bit-exact).

A run of few histories gives its gangs fewer slots than threads, ragged last gangs and claims
that run dry; a run of more histories than slots refills them.  Sums are integers, so images,
squares and counters equal the oracle's whatever the launch shape.
"""

import numpy as np
import pytest

from opengate_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,n,opts", [
    (32, 1, {}), (32, 31, {}), (32, 33, {}),
    (32, 152 * 32 + 1, {}),                                # one more history than a warp per SM
    (32, 152 * 640 + 77, dict(chunk=1)),                   # a full block, claims of the smallest size
    (32, 9001, dict(block_size=96, blocks_per_sm=1)),      # a gang of three warps
    (32, 5003, dict(block_size=160)),                      # a second gang of one warp
    (64, 1, {}), (64, 152 * 96 + 5, {}), (64, 700, dict(block_size=32)),
])
def test_pool_edges_bit_exact(built_lib, precision, n, opts):
    from opengate_gb300.engine import DoseEngine
    from oracle import oracle as O

    scene, _ = W.ct_phantom(shape=(40, 64, 64), spacing=4.8)
    with DoseEngine(scene, precision=precision, batch=1 << 20, **opts) as eng:
        eng.run(n, 97, 5)
        got = eng.edep(), eng.edep_squared(), eng.counters()
    ref = O.run_dose(scene, n, 97, first=5, batch=1 << 20, threads=4, precision=precision)
    assert got[2] == ref[2]
    assert np.array_equal(got[0], ref[0]) and np.array_equal(got[1], ref[1])


@pytest.mark.parametrize("mode", ["plain", "split", "forced"])
@pytest.mark.parametrize("precision,n,opts", [(32, 1, {}), (32, 2433, dict(chunk=1)), (32, 977, dict(block_size=96)),
                                              (64, 311, {})])
def test_phantom_stage_edges_bit_exact(built_lib, mode, precision, n, opts):
    """The SPECT phantom stage at the same edges: analog, with split requests, and the primary
    free flight that checks one record per thread."""
    import copy

    from opengate_gb300 import _capi as C
    from opengate_gb300.engine import SpectEngine
    from oracle import oracle as O

    scene, sp, _ = W.spect_phantom(shape=(20, 32, 32), spacing=9.6, n_runs=3)
    if mode == "split":
        sp.set_scatter_splitting(6, 3, 2, angle_tolerance_max=0.5)
    if mode == "forced":
        sp.set_free_flight()
        src = copy.copy(scene.source)
        src.dir_type, src.fd_angle_min, src.fd_angle_max = C.GG_DIR_FORCED, 0.0, 0.4
        scene.set_source(src)
    with SpectEngine(scene, sp, precision=precision, **opts) as eng:
        eng.run(n, 41)
        got = (eng.projection(),) if mode == "plain" else eng.weighted_projection(squared=True)
        cnt = eng.counters()
    run = O.run_spect if mode == "plain" else O.run_spect_ff
    *ref, rcnt = run(scene, sp, n, seed=41, threads=4, precision=precision)
    assert cnt == rcnt
    assert all(np.array_equal(a, b) for a, b in zip(got, ref))
