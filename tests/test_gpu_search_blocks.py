"""The search over 2 x 2 blocks of rays: neighbour indices against the oracle.

Odd images (blocks cut by the border), LOS lengths around the 64-sample segment and
its parts, clouds too dense for a part's candidates, a regular grid (equal
distances everywhere: the lowest original index wins), small boxes, and ray
tiles of odd sides, which are searched one ray per warp.  Indices are whole
numbers: every one must be equal.
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


def _loop():
    return synth.loop_snapshot(32, seed=3)


def _clumps():
    """Background plus clumps 30 times denser along each axis."""
    s = synth.loop_snapshot(24, seed=4)
    rng = np.random.default_rng(4)
    at = rng.integers(0, s.npoints, 6)
    pick = rng.integers(0, 6, 9000)
    new = [np.concatenate([a, a[at][pick] + rng.normal(0, 0.02, 9000).astype(np.float32)]) for a in (s.x, s.y, s.z)]
    rest = [np.concatenate([a, a[rng.integers(0, s.npoints, 9000)]]) for a in (s.n, s.T, s.vx, s.vy, s.vz)]
    return synth.Snapshot(*[np.ascontiguousarray(a, np.float32) for a in new + rest])


def _regular():
    return synth.loop_snapshot(33, seed=5, half_width=4.0, jitter=0.0)


def _check(ctx, s, nx, ny, nz, l, b):
    t = synth.line_table()
    eps, w = oracle.emission(s, t)
    sid, tid = ctx.snapshot(s), ctx.table(t)
    width = 1e5
    _, idx, _ = ctx.render(ctx.request(sid, tid, fg.METHOD_NN, nx, ny, nz, 4, l, b, width), want_idx=True)
    _, want, _ = oracle.nn_render(s, eps, w, t.lambda0, l, b, nx, ny, nz, 4, width, want_idx=True)
    np.testing.assert_array_equal(idx, want)
    ctx.drop_snapshot(sid)


@pytest.mark.parametrize("nx,ny,nz", [(101, 97, 63), (100, 97, 64), (97, 100, 65), (90, 91, 127), (89, 83, 129), (131, 129, 33),
                                      (300, 301, 9)])
def test_sizes(ctx, nx, ny, nz):
    _check(ctx, _loop(), nx, ny, nz, 0.4, -0.3)


@pytest.mark.parametrize("l,b", [(0.0, 0.0), (np.pi / 2, 0.0), (0.3, 1.2)])
def test_directions(ctx, l, b):
    _check(ctx, _loop(), 96, 93, 80, l, b)


@pytest.mark.parametrize("nz", [40, 300])
def test_dense_clumps(ctx, nz):
    _check(ctx, _clumps(), 150, 149, nz, 0.5, 0.2)


@pytest.mark.parametrize("n,l,b", [(129, 0.0, 0.0), (129, np.pi / 2, 0.0), (97, 0.4, 0.2)])
def test_equal_distances(ctx, n, l, b):
    _check(ctx, _regular(), n, n, n, l, b)


@pytest.mark.parametrize("tile", [(3, 5), (32, 1), (2, 2), (16, 4)])
def test_tiles(ctx, tile):
    ctx.set_march_config(*tile)
    try:
        _check(ctx, _loop(), 99, 98, 70, 0.4, -0.3)
    finally:
        ctx.set_march_config(0, 0)
