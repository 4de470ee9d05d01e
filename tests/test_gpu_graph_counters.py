"""Search counters switched on and off between replays of one batch's graph: a replay counts when they are on, and never into
memory that was given back when they were switched off."""

import numpy as np
import pytest

import fomo_gb300 as fg
from fomo_gb300 import synth

pytestmark = pytest.mark.gpu


def test_counters_and_replays():
    import torch

    with fg.Context(0) as ctx:
        sid, tid = ctx.snapshot(synth.loop_snapshot(20, seed=1)), ctx.table(synth.line_table())
        reqs = [ctx.request(sid, tid, fg.METHOD_NN, 24, 20, 70, 8, l, 0.2, 1.5e5) for l in (0.1, 0.7)]
        outs = [torch.empty(24 * 20 * 8, dtype=torch.float32, device="cuda:0") for _ in reqs]
        cubes = []
        for counters in (False, True, False, True, True):
            ctx.set_profiling(False, counters)
            ctx.render_batch_device(reqs, [o.data_ptr() for o in outs], graph=True)
            ctx.synchronize()
            assert ctx.profile_read()[1]["samples"] == (len(reqs) * 24 * 20 * 70 if counters else 0)
            cubes.append([o.cpu().numpy() for o in outs])
    for c in cubes[1:]:
        for a, b in zip(c, cubes[0]):
            np.testing.assert_array_equal(a, b)
