"""Split copies settled by approximate arithmetic, against the CPU oracle (bit-exact).

The split kernel rejects, drops or discards most copies from approximate trials and decides the
others exactly; every decision, hence every weight and counter, must be the exact sequence's - at
energies where the Compton angle is ill-conditioned, for cones the copies graze, for directions
along an axis of the scattering frame, and when a warp has fewer requests than lanes.
"""

import copy

import numpy as np
import pytest

from opengate_gb300 import _capi as C
from opengate_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("energy,angle,copies,along_z,precision", [
    (0.015, 0.2, 300, False, 32), (0.06, 0.02, 128, False, 32), (0.1405, 1.2, 33, False, 32),
    (1.0, 0.17, 64, False, 32), (0.3, 0.4, 40, True, 32), (0.2, 0.0, 7, False, 32), (0.0305, 0.17, 50, False, 64),
])
def test_split_copies_bit_exact(built_lib, energy, angle, copies, along_z, precision):
    from opengate_gb300.engine import SpectEngine
    from oracle import oracle as O

    scene, sp, _ = W.spect_phantom(shape=(20, 32, 32), spacing=9.6, n_runs=3)
    src = copy.copy(scene.source)
    src.ene_type, src.mono = C.GG_ENE_MONO, energy
    if along_z:
        src.dir_type, src.momentum = C.GG_DIR_MOMENTUM, [0.0, 0.0, -1.0]
    scene.set_source(src)
    sp.windows = [(0.001, 1.1), (0.5 * energy, energy)]
    sp.set_scatter_splitting(copies, 3, 4, angle_tolerance_max=angle)
    n = 4000
    with SpectEngine(scene, sp, precision=precision) as eng:
        eng.run(n, 83)
        w, w2 = eng.weighted_projection(squared=True)
        cnt = eng.counters()
    rw, rw2, rcnt = O.run_spect_ff(scene, sp, n, seed=83, threads=8, precision=precision)
    assert cnt == rcnt
    assert np.array_equal(w, rw) and np.array_equal(w2, rw2)
    assert cnt["world_steps"] > n
