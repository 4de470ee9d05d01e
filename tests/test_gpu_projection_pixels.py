"""The projection by pixel (many points) against the oracle's FP64 sums.

Images so small that a pixel's points are summed in pieces, images with more
pixels than points per warp batch and empty ones, bin counts around a 32-bin
window, one to four lines, and a cloud whose points mostly share a few pixels.

TOL: as a spectrum's values are (tests/test_gpu_emission_pass.py): 2 log n rounded to
FP32 (2.2e-6 of 10^x), one ulp of log10 (4.4e-6 of n^2), about 1e-6 for the profile
and the sums: below 1e-5 of the cube's maximum.
"""

import numpy as np
import pytest

import fomo_gb300 as fg
import oracle
from fomo_gb300 import synth
from tests import _golden as G

pytestmark = pytest.mark.gpu

TOL = 1e-5
LINES = ((5.8, 171.073), (6.0, 193.509), (6.2, 211.317), (6.4, 284.163))


@pytest.fixture(scope="module")
def clouds():
    with fg.Context(0) as ctx:
        loop, rope = synth.loop_snapshot(100, seed=8), synth.flux_rope_snapshot(950_000, seed=8)
        tabs = [synth.line_table(peak_logT=p, lambda0=lam) for p, lam in LINES]
        yield {"ctx": ctx, "tabs": tabs, "tids": [ctx.table(t) for t in tabs],
               "loop": (loop, ctx.snapshot(loop)), "rope": (rope, ctx.snapshot(rope))}


@pytest.mark.parametrize("cloud,nx,ny,L,nl,l,b", [
    ("loop", 7, 9, 33, 1, 0.3, 0.2), ("loop", 33, 31, 32, 2, 0.0, 0.0), ("loop", 257, 255, 31, 1, 1.1, -0.3),
    ("loop", 90, 64, 65, 4, 0.3, 0.2), ("loop", 64, 50, 129, 1, 0.5, 0.1), ("loop", 50, 64, 97, 3, 0.5, 0.1),
    ("rope", 24, 24, 40, 2, 0.0, 0.0), ("rope", 700, 500, 2, 1, 0.4, 0.3)])
def test_spectra(clouds, cloud, nx, ny, L, nl, l, b):
    ctx = clouds["ctx"]
    s, sid = clouds[cloud]
    width = 3.1e5
    reqs = [ctx.request(sid, t, fg.METHOD_PROJECTION, nx, ny, 64, L, l, b, width) for t in clouds["tids"][:nl]]
    cubes, infos = ctx.render_batch(reqs)
    for t, cube in zip(clouds["tabs"], cubes):
        eps, w = oracle.emission(s, t)
        want, _, view = oracle.projection_render(s, eps, w, t.lambda0, l, b, nx, ny, 64, L, width)
        assert G.norm_max_err(cube.ravel(), want.ravel()) <= TOL
    assert (infos[0].minx, infos[0].maxx) == (view[0], view[1])


def test_views_of_one_batch_and_a_replayed_one(clouds):
    """Several views share the lists' memory; a graph replayed with other outputs fills those."""
    torch = pytest.importorskip("torch")
    ctx = clouds["ctx"]
    _, sid = clouds["loop"]
    reqs = [ctx.request(sid, clouds["tids"][0], fg.METHOD_PROJECTION, nx, 40, 64, 32, l, 0.1, 3.1e5)
            for nx, l in ((40, 0.1), (90, 0.7), (61, 1.2))]
    alone = [ctx.render(q)[0] for q in reqs]
    for _ in range(2):
        outs = [torch.full((q.ny, q.nx, q.nlambda), 7.0, device="cuda") for q in reqs]
        torch.cuda.synchronize()
        ctx.render_batch_device(reqs, [o.data_ptr() for o in outs], graph=True)
        ctx.synchronize()
        for o, want in zip(outs, alone):
            # the points of a pixel are summed in another order: FP32 sums with compensation
            assert G.norm_max_err(o.cpu().numpy().ravel(), want.ravel()) <= 1e-6
