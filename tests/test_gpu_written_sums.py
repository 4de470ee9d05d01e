"""The written spectra are the sums times the view's scale, rounded once.

The same sums are written with two scales (a table in DN units carries the pixel's solid angle); both are known in FP64, so
the ratio of the two cubes is theirs within two roundings to FP32 of 2^-24 each.  Abundances move the values from where
FP32 pairs form them down to where the FP64 expression does (below 1e-30).
"""

import dataclasses

import numpy as np
import pytest

import fomo_gb300 as fg
from fomo_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("method", [fg.METHOD_NN, fg.METHOD_PROJECTION])
@pytest.mark.parametrize("abund", [1e-16, 1e-8, 1.0, 1e12])
@pytest.mark.parametrize("nlam", [7, 33, 130])
def test_two_scales(method, abund, nlam):
    s, t = synth.loop_snapshot(100, seed=3), synth.line_table()
    with fg.Context(0) as ctx:
        sid = ctx.snapshot(s)
        cubes, scales = [], []
        for table in (t, dataclasses.replace(t, unit=t.unit + " DN")):
            req = ctx.request(sid, ctx.table(table), method, 40, 37, 80, nlam, 0.4, 0.2, 1.5e5, abund)
            cube, _, info = ctx.render(req)
            cubes.append(cube.astype(np.float64))
            scales.append(info.scale)
    assert scales[0] != scales[1]
    normal = np.minimum(cubes[0], cubes[1]) > 1.2e-38
    assert normal.any() and ((cubes[0] > 0) | (cubes[1] == 0)).all()
    ratio = cubes[0][normal] / cubes[1][normal] * (scales[1] / scales[0])
    # the projection's sums vary by their order where pixels are summed in pieces or by atomics (none here: 676 points a pixel
    # make two pieces of one pixel's sum, each rounded)
    assert np.abs(ratio - 1).max() <= (2 if method == fg.METHOD_NN else 64) * 2.0**-24 * 1.01
