"""fomo_render_noalloc searches as a regular render does: the same gather radius, and so the same samples left to
the lane walks.

Its first pass takes the same 64-sample segments as the regular search of one ray per warp (ray tiles of odd sides), so
every counter of that search is equal whatever the order of the rays; the counters are whole numbers.
"""

import ctypes

import pytest

import fomo_gb300 as fg
from fomo_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cloud", ["uniform", "clustered"])
@pytest.mark.parametrize("nx,ny,nz,nlam", [(33, 20, 65, 8), (64, 61, 200, 1), (96, 96, 256, 16)])
def test_same_samples_left_open(cloud, nx, ny, nz, nlam):
    import torch

    s = synth.loop_snapshot(40, seed=2) if cloud == "uniform" else synth.flux_rope_snapshot(60000, seed=2)
    t = synth.line_table() if nlam > 1 else synth.broadband_table(171)
    with fg.Context(0) as ctx:
        req = ctx.request(ctx.snapshot(s), ctx.table(t), fg.METHOD_NN, nx, ny, nz, nlam, 0.4, 0.3, 1.5e5)
        out = torch.empty(nx * ny * nlam, dtype=torch.float32, device="cuda:0")
        ctx.set_march_config(3, 5)
        ctx.render_device(req, out.data_ptr())  # the emissivity is resident from here on
        ctx.synchronize()
        ctx.set_profiling(False, True)
        ctx.render_device(req, out.data_ptr())
        regular = ctx.profile_read()[1]
        rc = fg.lib().fomo_render_noalloc(ctx.h, ctypes.byref(req), ctypes.c_void_p(out.data_ptr()), None)
        assert rc == fg.OK
        noalloc = ctx.profile_read()[1]
    for k in ("samples", "segments", "candidates", "scanned", "not_gathered", "fallbacks"):
        assert noalloc[k] == regular[k], (k, noalloc[k], regular[k])
