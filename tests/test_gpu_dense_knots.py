"""A cloud that fills its box evenly, with a few dense knots in it: few empty cells, and some with thousands of points.

Samples near a knot that the search leaves open must not be one lane's walk through a whole knot: the hard queue takes them
(a counter above zero), in narrow-box views too.  The neighbours are the oracle's, every one.
"""

import numpy as np
import pytest

import fomo_gb300 as fg
import oracle
from fomo_gb300 import synth

pytestmark = pytest.mark.gpu


def _knots(side, share, seed):
    s = synth.loop_snapshot(side, seed=seed)
    rng = np.random.default_rng(seed)
    m = int(share * s.npoints)
    at, pick = rng.integers(0, s.npoints, 8), rng.integers(0, 8, m)
    new = [np.concatenate([a, a[at][pick] + rng.normal(0, 0.03, m).astype(np.float32)]) for a in (s.x, s.y, s.z)]
    rest = [np.concatenate([a, a[rng.integers(0, s.npoints, m)]]) for a in (s.n, s.T, s.vx, s.vy, s.vz)]
    return synth.Snapshot(*[np.ascontiguousarray(a, np.float32) for a in new + rest])


@pytest.mark.parametrize("share", [0.0, 0.1])
@pytest.mark.parametrize("nx,ny,nz", [(100, 101, 129), (128, 64, 300)])
def test_knots(share, nx, ny, nz):
    s = _knots(40, share, seed=3)
    t = synth.line_table()
    eps, w = oracle.emission(s, t)
    with fg.Context(0) as ctx:
        req = ctx.request(ctx.snapshot(s), ctx.table(t), fg.METHOD_NN, nx, ny, nz, 4, 0.5, 0.2, 1e5)
        ctx.set_profiling(False, True)
        _, idx, _ = ctx.render(req, want_idx=True)
        hard = ctx.profile_read()[1]["hard"]
    _, want, _ = oracle.nn_render(s, eps, w, t.lambda0, 0.5, 0.2, nx, ny, nz, 4, 1e5, want_idx=True)
    np.testing.assert_array_equal(idx, want)
    assert (hard > 0) == (share > 0)
