"""Projections fetched as FP64 (converted on the device) against NumPy's conversion of the same words."""

import numpy as np
import pytest

from opengate_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size,runs", [((1, 1), 1), ((7, 5), 3), ((33, 64), 2)])
def test_weighted_projection_matches_host_conversion(built_lib, size, runs):
    from opengate_gb300.engine import SpectEngine

    scene, sp, _ = W.spect_phantom(shape=(20, 32, 32), spacing=9.6, n_runs=runs)
    sp.size, sp.spacing = list(size), [565.76 / size[0], 565.76 / size[1]]
    sp.set_free_flight()
    with SpectEngine(scene, sp) as eng:
        eng.record_singles(400_000)
        eng.run(40_000 // runs, 11)
        w, w2 = eng.weighted_projection(squared=True)
        counts, singles = eng.projection(), eng.singles()
    assert len(singles) and counts.sum() == 0  # weighted mode: no counts
    # the fixed-point sums of the listed singles, as the digitizer makes them (2^-32 units)
    ref, ref2 = np.zeros_like(w), np.zeros_like(w)
    half = [0.5 * n * s for n, s in zip(sp.size, sp.spacing)]
    q = np.rint(np.float32(singles["weight"]) * np.float32(2.0 ** 32)).astype(np.uint64)
    x = np.float32(np.float32(singles["a1"]) + np.float32(half[0])) * np.float32(1 / sp.spacing[0])
    y = np.float32(np.float32(singles["a2"]) + np.float32(half[1])) * np.float32(1 / sp.spacing[1])
    words, squares = {}, {}
    for k, (lo, hi) in enumerate(sp.windows):
        e = singles["energy"]
        for i in np.flatnonzero((e >= np.float32(lo)) & (e < np.float32(hi))):
            if 0 <= x[i] < sp.size[0] and 0 <= y[i] < sp.size[1]:
                at = (singles["head"][i], singles["run"][i] * sp.n_windows + k, int(y[i]), int(x[i]))
                words[at] = words.get(at, 0) + int(q[i])
                squares.setdefault(at, []).append(int(q[i]) ** 2)
    for at, v in words.items():
        ref[at] = float(v) * 2.0 ** -32
        lo = float(sum(s & 0xffffffff for s in squares[at])) * 2.0 ** -64
        ref2[at] = float(sum(s >> 32 for s in squares[at])) * 2.0 ** -32 + lo
    assert np.array_equal(w, ref) and np.array_equal(w2, ref2)
