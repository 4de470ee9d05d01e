"""Infinite emissivities: a sum that holds one is infinite, as the reference's plain sum is, and not NaN.

n^2 overflows FP32 for n > 1.8e19, so a table whose density axis reaches there gives points of infinite emissivity.  Some
rays meet them early and go on through finite ones, some meet them last, most none.  The lambda range is so narrow that no
profile of an infinite peak underflows to 0 (infinity times 0 is NaN in any order): |2 d / w|^2 < 100.  Which elements are
infinite, and that none is NaN, must agree with the oracle; finite ones within the usual 1e-4 of the largest.
"""

import dataclasses

import numpy as np
import pytest

import fomo_gb300 as fg
import oracle
from fomo_gb300 import synth

pytestmark = pytest.mark.gpu


def _case(side, imaging):
    s = synth.loop_snapshot(side, seed=5)
    n = s.n.copy()
    rng = np.random.default_rng(5)
    low, high = s.z < -3.0, s.z > 4.0
    edge = (np.abs(s.x) < 1.5) & (np.abs(s.y) < 1.5)
    n[(low | high) & edge & (rng.random(s.npoints) < 0.3)] = 1e20
    s = dataclasses.replace(s, n=n)
    t = synth.broadband_table(171) if imaging else synth.line_table()
    logn = np.linspace(8.0, 21.0, t.nrho).astype(np.float32)
    return s, dataclasses.replace(t, logn=logn)


def _same(got, want):
    assert np.isinf(want).any() and np.isfinite(want).any() and not np.isnan(want).any()
    np.testing.assert_array_equal(np.isinf(got), np.isinf(want))
    f = np.isfinite(want)
    assert np.isfinite(got[f]).all()
    assert np.abs(got[f].astype(np.float64) - want[f]).max() <= 1e-4 * np.abs(want[f]).max()


@pytest.mark.parametrize("nlam", [1, 12])
@pytest.mark.parametrize("nx,ny,nz", [(9, 7, 33), (24, 24, 96), (40, 40, 300)])
def test_render(nx, ny, nz, nlam):
    s, t = _case(24, nlam == 1)
    eps, w = oracle.emission(s, t, imaging=nlam == 1)
    assert np.isinf(eps).any()
    with fg.Context(0) as ctx:
        cube, _, _ = ctx.render(ctx.request(ctx.snapshot(s), ctx.table(t), fg.METHOD_NN, nx, ny, nz, nlam, 0.2, 0.1, 8e4))
    want, _, _ = oracle.nn_render(s, eps, w, t.lambda0, 0.2, 0.1, nx, ny, nz, nlam, 8e4, is_dn=t.is_dn)
    _same(cube, want)


@pytest.mark.parametrize("side", [24, 100])  # few points: added one by one; many: by pixel
def test_projection(side):
    s, t = _case(side, False)
    eps, w = oracle.emission(s, t)
    with fg.Context(0) as ctx:
        cube, _, _ = ctx.render(ctx.request(ctx.snapshot(s), ctx.table(t), fg.METHOD_PROJECTION, 30, 28, 1, 12, 0.2, 0.1, 8e4))
    want = oracle.projection_render(s, eps, w, t.lambda0, 0.2, 0.1, 30, 28, 1, 12, 8e4)
    _same(cube, want[0] if isinstance(want, tuple) else want)
