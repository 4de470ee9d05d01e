"""Samples queued for whole warps: not more than the warps can take at once."""

import numpy as np
import pytest

import fomo_gb300 as fg
import oracle
from fomo_gb300 import synth

pytestmark = pytest.mark.gpu


def _knots(side, share, seed, width):
    s = synth.loop_snapshot(side, seed=seed)
    rng = np.random.default_rng(seed)
    m = int(share * s.npoints)
    at, pick = rng.integers(0, s.npoints, 8), rng.integers(0, 8, m)
    new = [np.concatenate([a, a[at][pick] + rng.normal(0, width, m).astype(np.float32)]) for a in (s.x, s.y, s.z)]
    rest = [np.concatenate([a, a[rng.integers(0, s.npoints, m)]]) for a in (s.n, s.T, s.vx, s.vy, s.vz)]
    return synth.Snapshot(*[np.ascontiguousarray(a, np.float32) for a in new + rest])


def test_long_hard_queue():
    """Wide knots seen in a small image: most of the open samples lie in dense cells.  Once 8,192 samples are queued a
    lane's walk has the longer budget (192, at which 1,700 of these samples are hard): each of the 152 x 32 warps adds at
    most 32 samples more before it sees that.  With the short budget throughout 281,000 are queued."""
    s = _knots(64, 0.3, seed=3, width=0.5)
    t = synth.line_table()
    eps, w = oracle.emission(s, t)
    with fg.Context(0) as ctx:
        req = ctx.request(ctx.snapshot(s), ctx.table(t), fg.METHOD_NN, 101, 102, 300, 4, 0.5, 0.2, 1e5)
        ctx.set_profiling(False, True)
        _, idx, _ = ctx.render(req, want_idx=True)
        hard = ctx.profile_read()[1]["hard"]
    _, want, _ = oracle.nn_render(s, eps, w, t.lambda0, 0.5, 0.2, 101, 102, 300, 4, 1e5, want_idx=True)
    np.testing.assert_array_equal(idx, want)
    assert hard <= 8192 + 32 * 32 * 152 + 1700
