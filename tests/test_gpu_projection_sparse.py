"""Projections of images with few points a pixel go by the direct kernel (no lists in memory), with more by pixel; both sides of
the line against the oracle.  TOL as in tests/test_gpu_projection_pixels.py: below 1e-5 of the cube's maximum."""

import numpy as np
import pytest

import fomo_gb300 as fg
import oracle
from fomo_gb300 import synth

pytestmark = pytest.mark.gpu

N = 80**3  # x 1 line x 64 bins, and x 2: above 900,000 points x lines x windows


@pytest.mark.parametrize("lines,per_pixel", [(1, 0.5), (1, 3.9), (1, 4.1), (2, 0.5), (2, 2.9), (2, 3.1)])
def test_few_points_a_pixel(lines, per_pixel):
    import torch

    s = synth.loop_snapshot(80, seed=4)
    tabs = [synth.line_table(peak_logT=p, lambda0=lam) for p, lam in ((5.8, 171.073), (6.0, 193.509))[:lines]]
    nx = int(round((N / per_pixel) ** 0.5))
    ny = int(round(N / per_pixel / nx))
    outs = [torch.empty((ny, nx, 64), dtype=torch.float32, device="cuda:0") for _ in tabs]
    with fg.Context(0) as ctx:
        sid = ctx.snapshot(s)
        tids = [ctx.table(t) for t in tabs]
        # the emissivities are resident from here on, and a little working memory
        small = torch.empty(8 * 8 * 4 * lines, dtype=torch.float32, device="cuda:0")
        ctx.render_batch_device([ctx.request(sid, t, fg.METHOD_NN, 8, 8, 4, 4, 0.3, 0.2, 1.5e5) for t in tids],
                                [small.data_ptr() + 1024 * k for k in range(lines)])
        before = ctx.memory()[0]
        reqs = [ctx.request(sid, t, fg.METHOD_PROJECTION, nx, ny, 1, 64, 0.3, 0.2, 1.5e5) for t in tids]
        ctx.render_batch_device(reqs, [o.data_ptr() for o in outs])
        ctx.synchronize()
        taken = ctx.memory()[0] - before
        cubes = [o.cpu().numpy() for o in outs]
    # without lists 24 bytes of queues a pixel of the 8 x 4 tiles and some tables; the lists take 12 bytes a point more
    queues = 24 * (-(-nx // 8) * 8) * (-(-ny // 4) * 4)
    assert (taken > queues + 6 * N) == (per_pixel > (4 if lines == 1 else 3)), taken
    for t, cube in zip(tabs, cubes):
        eps, w = oracle.emission(s, t)
        want, _, _ = oracle.projection_render(s, eps, w, t.lambda0, 0.3, 0.2, nx, ny, 1, 64, 1.5e5)
        assert np.abs(cube - want).max() <= 1e-5 * np.abs(want).max()
