"""The list of a dose grid that scores edep and dose, against the CPU oracle (bit-exact).

Fine grids give every interaction its own voxel, so lists fill and are flushed inside a history;
coarse ones merge the deposits; launches of one warp and of full blocks.
"""

import numpy as np
import pytest

from opengate_gb300 import _capi as C
from opengate_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,n,voxel,opts", [
    (32, 33, 1.5, {}), (32, 152 * 640 + 7, 1.5, {}), (32, 5003, 100.0, dict(block_size=32)),
    (64, 4001, 1.5, {}), (64, 401, 25.0, dict(block_size=96)),
])
def test_edep_and_dose_lists_bit_exact(built_lib, precision, n, voxel, opts):
    from opengate_gb300.engine import DoseEngine
    from oracle import oracle as O

    scene, _ = W.ct_phantom(shape=(40, 64, 64), spacing=4.8)
    g = C.DoseGridDesc()
    g.dims[:] = [max(1, int(d * 4.8 / voxel)) for d in (64, 64, 40)]
    g.spacing[:] = [voxel] * 3
    g.corner[:] = scene.corner
    g.score_dose = 1
    with DoseEngine(scene, precision=precision, batch=1 << 20, **opts) as e:
        e.set_dose_grid(list(g.dims), list(g.spacing), list(g.corner))
        e.run(n, 17)
        got = (e.edep(), e.edep_squared(), e.dose_sum(), e.dose_sum_squared()), e.counters()
    *ref, cnt = O.run_dose_grid(scene, g, n, 17, threads=8, precision=precision, batch=1 << 20)
    assert got[1] == cnt
    for a, b in zip(got[0], ref):
        assert np.array_equal(a, b)
    if n > 1000 and voxel < 10.0:
        assert cnt["list_overflows"] > 0
