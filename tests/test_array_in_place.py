"""Device arrays of a snapshot: read where they are only if aligned for 32-bit loads and whole in their allocation."""

import os
import shutil
import subprocess

import numpy as np
import pytest

import fomo_gb300 as fg
from fomo_gb300 import synth

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_rule(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    exe = str(tmp_path / "array_in_place")
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-I" + os.path.join(ROOT, "fomo_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "array_in_place.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


@pytest.mark.gpu
@pytest.mark.parametrize("shift", [1, 2, 3, 4])
def test_arrays_at_any_byte(shift):
    import torch

    s, t = synth.loop_snapshot(13, seed=1), synth.line_table()
    raw = []
    for a in s.arrays():
        d = torch.empty(a.nbytes + 8, dtype=torch.uint8, device="cuda:0")
        d[shift:shift + a.nbytes] = torch.from_numpy(np.ascontiguousarray(a).view(np.uint8)).cuda()
        raw.append(d)
    torch.cuda.synchronize()
    with fg.Context(0) as ctx:
        tid = ctx.table(t)
        ids = ctx.snapshot(s), ctx.snapshot_device(s.npoints, [d.data_ptr() + shift for d in raw])
        got = [ctx.render(ctx.request(sid, tid, fg.METHOD_NN, 20, 17, 40, 8, 0.3, 0.2, 1.5e5), want_idx=True)[:2] for sid in ids]
    np.testing.assert_array_equal(got[0][1], got[1][1])
    np.testing.assert_array_equal(got[0][0], got[1][0])
