"""The emission pass at the edges of its batches.

A ray's runs of equal neighbours are collected 128 samples at a time, binned 32
at a time, and each line's lambda bins in windows of 32.  LOS lengths and bin
counts around those sizes, one to four lines, imaging and Thomson, against the
FP64 oracle on the same neighbours.

TOL: FP32 arithmetic of eps = k 10^(2 log n) G / w.  The exponent 2 log n lies in
[16, 32), half an ulp 9.5e-7 or 2.2e-6 of 10^x; log10 may differ by one ulp from
the host's (4.4e-6 for n^2); the Gaussian's exponent and the sums add about 1e-6.
Together below 1e-5 of a value, and of the cube's maximum.
"""

import numpy as np
import pytest

import fomo_gb300 as fg
import oracle
from fomo_gb300 import synth
from tests import _golden as G

pytestmark = pytest.mark.gpu

TOL = 1e-5
WIDTH = 3.1e5  # m/s: more than one window of bins around the line


@pytest.fixture(scope="module")
def ctx():
    with fg.Context(0) as c:
        yield c


@pytest.mark.parametrize("nz,L,nlines", [(2, 2, 1), (31, 32, 1), (32, 33, 2), (33, 31, 3), (127, 64, 4), (128, 65, 4),
                                         (129, 97, 2), (160, 128, 3), (161, 128, 4), (257, 129, 1), (300, 256, 1)])
def test_spectra(ctx, nz, L, nlines):
    s = synth.loop_snapshot(20, seed=nz)
    lines = [(5.8, 171.073), (6.0, 193.509), (6.2, 211.317), (6.4, 284.163)][:nlines]
    tabs = [synth.line_table(peak_logT=p, lambda0=lam) for p, lam in lines]
    sid = ctx.snapshot(s)
    tids = [ctx.table(t) for t in tabs]
    l, b = 0.3, -0.2
    reqs = [ctx.request(sid, t, fg.METHOD_NN, 13, 11, nz, L, l, b, WIDTH) for t in tids]
    cubes, _ = ctx.render_batch(reqs)
    for t, cube in zip(tabs, cubes):
        eps, w = oracle.emission(s, t)
        want, _, _ = oracle.nn_render(s, eps, w, t.lambda0, l, b, 13, 11, nz, L, WIDTH)
        assert G.norm_max_err(cube.ravel(), want.ravel()) <= TOL
    ctx.drop_snapshot(sid)


@pytest.mark.parametrize("nz,nch", [(2, 1), (32, 2), (33, 3), (128, 6), (129, 8), (300, 5)])
def test_channels(ctx, nz, nch):
    s = synth.flux_rope_snapshot(20000, seed=nz)
    tabs = [synth.broadband_table(100 + 20 * k, peak_logT=5.8 + 0.08 * k) for k in range(nch)]
    sid = ctx.snapshot(s)
    reqs = [ctx.request(sid, ctx.table(t), fg.METHOD_NN, 13, 11, nz, 1, 0.5, 0.3, 1e5) for t in tabs]
    cubes, _ = ctx.render_batch(reqs)
    for t, cube in zip(tabs, cubes):
        eps, w = oracle.emission(s, t, imaging=True)
        want, _, _ = oracle.nn_render(s, eps, w, t.lambda0, 0.5, 0.3, 13, 11, nz, 1, 1e5, is_dn=True)
        assert G.norm_max_err(cube.ravel(), want.ravel()) <= TOL
    ctx.drop_snapshot(sid)


@pytest.mark.parametrize("nz", [2, 33, 128, 257])
def test_thomson(ctx, nz):
    s = synth.thomson_snapshot(20, seed=nz)
    tot, pol = oracle.thomson_emission(s)
    sid = ctx.snapshot(s)
    cube, _, _ = ctx.render(ctx.request(sid, 0, fg.METHOD_THOMSON, 13, 11, nz, 1, 0.2, 0.1, 1e5))
    want, _, _ = oracle.thomson_render(s, tot, pol, 0.2, 0.1, 13, 11, nz)
    assert G.norm_max_err(cube.ravel(), want.ravel()) <= TOL
    ctx.drop_snapshot(sid)
