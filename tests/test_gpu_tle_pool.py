"""The track-length estimator's walks at the edges of their rounds, against the CPU oracle (bit-exact).

Paths of fewer and more boundaries than a round walks, lists that fill in the middle of one,
photons above the threshold between scored ones, a beam whose photons share their voxels and
one whose photons do not, launches of one warp and of full blocks.
"""

import copy

import numpy as np
import pytest

from opengate_gb300 import _capi as C
from opengate_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scene,precision,n,tle,opts", [
    ("pencil", 32, 1, (np.inf, 0.0, "EPDL"), {}),
    ("pencil", 32, 152 * 640 + 33, (np.inf, 0.0, "EPDL"), {}),
    ("pencil", 32, 4001, (0.25, 0.05, "NIST"), dict(block_size=96)),     # scored after the first scatter
    ("pencil", 64, 1501, (0.25, 0.05, "NIST"), {}),
    ("wide", 32, 20_011, (np.inf, 0.0, "EPDL"), dict(chunk=1)),
    ("ct", 32, 9001, (1.2, 0.04, "EPDL"), dict(block_size=32)),
    ("thin", 32, 5003, (np.inf, 0.0, "NIST"), {}),                       # paths of one to three voxels
    ("thin", 64, 701, (np.inf, 0.0, "NIST"), dict(block_size=32)),
])
def test_walks_bit_exact(built_lib, scene, precision, n, tle, opts):
    from opengate_gb300.engine import DoseEngine
    from oracle import oracle as O

    if scene == "ct":
        sc, _ = W.ct_phantom(shape=(40, 64, 64), spacing=4.8)
    elif scene == "thin":
        sc, _ = W.ct_phantom(shape=(2, 3, 3), spacing=60.0)
    else:
        sc = W.water_pencil(energy=0.3)
        if scene == "wide":
            src = copy.copy(sc.source)
            src.dir_type = C.GG_DIR_ISO
            sc.set_source(src)
    with DoseEngine(sc, precision=precision, batch=1 << 20, **opts) as eng:
        eng.set_tle(*tle)
        eng.run(n, 23, 11)
        got = eng.edep(), eng.edep_squared(), eng.counters()
    ref = O.run_dose(sc, n, 23, first=11, batch=1 << 20, threads=4, precision=precision, tle=sc.tle_desc(*tle))
    assert got[2] == ref[2]
    assert np.array_equal(got[0], ref[0]) and np.array_equal(got[1], ref[1])
