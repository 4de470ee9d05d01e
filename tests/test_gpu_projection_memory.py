"""A projection lists its points by pixel only where there is memory for the lists; without, the direct kernel renders it.

* a context whose budget holds everything but the lists renders the projection all the same;
* a server counts the lists in a request's admission bytes: with a budget for two requests without lists but for one with,
  the second starts after the first is done, and one whose lists exceed the budget alone goes without them.

Both kernels sum the same terms in FP32 in different orders; 1e-5 of the cube's largest value is 10 times the difference of
the sums' rounding (at most 20 terms of one sign that matter per bin, 2^-24 each).
"""

import numpy as np
import pytest

import fomo_gb300 as fg
from fomo_gb300 import synth

pytestmark = pytest.mark.gpu

NX, NY, NL = 200, 180, 64


def _request(sid, tid, l=0.3):
    return fg.Context.request(sid, tid, fg.METHOD_PROJECTION, NX, NY, 1, NL, l, 0.2, 1.5e5)


def _lists(n):
    return 12 * n  # a place and a list entry per point; the rest is below a tenth of that here


def _device_snapshot(ctx, s):
    import torch

    arrays = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in s.arrays()]
    torch.cuda.synchronize()
    return ctx.snapshot_device(s.npoints, [a.data_ptr() for a in arrays])


def _close(a, b):
    assert np.isfinite(a).all() and np.abs(a - b).max() <= 1e-5 * np.abs(b).max()


def test_tight_context():
    s, t = synth.loop_snapshot(110, seed=2), synth.line_table()
    with fg.Context(0) as ctx:
        sid, tid = _device_snapshot(ctx, s), ctx.table(t)
        ref, _, _ = ctx.render(_request(sid, tid))
        used = ctx.memory()[0]
    with fg.Context(0, hbm_budget=used - _lists(s.npoints) // 2) as ctx:
        sid, tid = _device_snapshot(ctx, s), ctx.table(t)
        for _ in range(2):
            cube, _, _ = ctx.render(_request(sid, tid))
            _close(cube, ref)


def _served(budget, s, t, refs):
    with fg.Server(0, hbm_budget=budget) as srv:
        sid, tid = srv.ctx.snapshot(s), srv.ctx.table(t)
        outs = [np.full((NY, NX, NL), np.nan, np.float32) for _ in refs]
        tickets = [srv.submit(_request(sid, tid, l), o) for l, o in zip((0.3, 0.9), outs)]
        stats = [srv.wait(k) for k in tickets]
    for o, r in zip(outs, refs):
        _close(o, r)
    return stats


def test_admission():
    s, t = synth.loop_snapshot(126, seed=2), synth.line_table()
    with fg.Context(0) as ctx:
        sid, tid = ctx.snapshot(s), ctx.table(t)
        refs = [ctx.render(_request(sid, tid, l))[0] for l in (0.3, 0.9)]
    base = 4 * NX * NY * NL + (1 << 21)  # the cube, its queues and tables (below 2 MB)
    first, second = _served(base + _lists(s.npoints) * 17 // 16 + base // 2, s, t, refs)
    assert second.t_start >= first.t_done
    _served(base + _lists(s.npoints) // 2, s, t, refs)
