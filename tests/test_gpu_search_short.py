"""Rays of few samples through a dense cloud, searched as blocks of rays: segments whose capsule overflows the candidate list
go to the lane walks up to 16 samples, to march_split's parts above.  Every neighbour index must be the oracle's."""

import numpy as np
import pytest

import fomo_gb300 as fg
import oracle
from fomo_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def cloud():
    return synth.loop_snapshot(64, seed=7)


@pytest.mark.parametrize("nz", [1, 2, 8, 15, 16, 17, 24])
@pytest.mark.parametrize("nx,ny", [(128, 129), (250, 96)])
def test_short_rays(cloud, nx, ny, nz):
    t = synth.line_table()
    eps, w = oracle.emission(cloud, t)
    with fg.Context(0) as ctx:
        req = ctx.request(ctx.snapshot(cloud), ctx.table(t), fg.METHOD_NN, nx, ny, nz, 4, 0.7, 0.3, 1e5)
        _, idx, _ = ctx.render(req, want_idx=True)
    _, want, _ = oracle.nn_render(cloud, eps, w, t.lambda0, 0.7, 0.3, nx, ny, nz, 4, 1e5, want_idx=True)
    np.testing.assert_array_equal(idx, want)
