"""An image of more columns than 65,535 blocks of 128 table entries, two rows of it: neighbours of the first row and its pixels
against the oracle."""

import numpy as np
import pytest

import fomo_gb300 as fg
import oracle
from fomo_gb300 import synth

pytestmark = pytest.mark.gpu


def test_wide_image():
    nx = 128 * 65535 + 3
    s, t = synth.loop_snapshot(8, seed=1), synth.broadband_table(171)
    eps, w = oracle.emission(s, t, imaging=True)
    with fg.Context(0) as ctx:
        req = ctx.request(ctx.snapshot(s), ctx.table(t), fg.METHOD_NN, nx, 2, 1, 1, 0.3, 0.2, 1e5)
        cube, idx, _ = ctx.render(req, want_idx=True)
    want, widx, _ = oracle.nn_render(s, eps, w, t.lambda0, 0.3, 0.2, nx, 2, 1, 1, 1e5, is_dn=t.is_dn, rows=(0, 1), want_idx=True)
    np.testing.assert_array_equal(idx[:1], widx)
    assert np.abs(cube[:1].astype(np.float64) - want).max() <= 1e-4 * np.abs(want).max()
