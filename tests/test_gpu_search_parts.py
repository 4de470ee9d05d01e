"""Rays cut into stretches of segments, and overflowing segments into halves: neighbour indices against the oracle.

Images of few rays (the smallest image, two rows, odd sides; ray tiles of odd sides, which are searched one ray per
warp), LOS lengths around whole numbers of 64-sample segments, and a cloud so dense that segments
overflow on either half.  Indices are whole numbers: every one must be equal.
"""

import numpy as np
import pytest

import fomo_gb300 as fg
import oracle
from fomo_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    with fg.Context(0) as c:
        yield c


def _clumps():
    """Background plus clumps of 1,500 points, narrower than a LOS segment is long."""
    s = synth.loop_snapshot(20, seed=8)
    rng = np.random.default_rng(8)
    at = rng.integers(0, s.npoints, 8)
    pick = rng.integers(0, 8, 12000)
    new = [np.concatenate([a, a[at][pick] + rng.normal(0, 0.03, 12000).astype(np.float32)]) for a in (s.x, s.y, s.z)]
    rest = [np.concatenate([a, a[rng.integers(0, s.npoints, 12000)]]) for a in (s.n, s.T, s.vx, s.vy, s.vz)]
    return synth.Snapshot(*[np.ascontiguousarray(a, np.float32) for a in new + rest])


def _check(ctx, s, nx, ny, nz, l, b):
    t = synth.line_table()
    eps, w = oracle.emission(s, t)
    sid, tid = ctx.snapshot(s), ctx.table(t)
    _, idx, _ = ctx.render(ctx.request(sid, tid, fg.METHOD_NN, nx, ny, nz, 4, l, b, 1e5), want_idx=True)
    _, want, _ = oracle.nn_render(s, eps, w, t.lambda0, l, b, nx, ny, nz, 4, 1e5, want_idx=True)
    np.testing.assert_array_equal(idx, want)
    ctx.drop_snapshot(sid)


@pytest.mark.parametrize("nz", [1, 63, 64, 65, 128, 129, 700])
@pytest.mark.parametrize("nx,ny", [(2, 2), (17, 2), (13, 31)])
@pytest.mark.parametrize("tile", [(0, 0), (3, 5)])
def test_few_rays(ctx, nx, ny, nz, tile):
    ctx.set_march_config(*tile)
    try:
        _check(ctx, synth.loop_snapshot(24, seed=6), nx, ny, nz, 0.4, -0.3)
    finally:
        ctx.set_march_config(0, 0)


@pytest.mark.parametrize("nx,ny,nz", [(40, 39, 33), (33, 40, 64), (31, 30, 97), (25, 24, 400)])
def test_overflow(ctx, nx, ny, nz):
    _check(ctx, _clumps(), nx, ny, nz, 0.5, 0.2)
