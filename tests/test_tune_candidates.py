"""What the autotuner measures includes what an untuned context runs."""

import os
import shutil
import subprocess

import pytest

import fomo_gb300 as fg
from fomo_gb300 import synth

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_candidates(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    exe = str(tmp_path / "tune_candidates")
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-I" + os.path.join(ROOT, "fomo_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "tune_candidates.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


@pytest.mark.gpu
def test_choice_is_a_candidate(tmp_path):
    cache = str(tmp_path / "tune.txt")
    with fg.Context(0) as ctx:
        sid, tid = ctx.snapshot(synth.flux_rope_snapshot(30000, seed=1)), ctx.table(synth.line_table())
        ctx.autotune([ctx.request(sid, tid, fg.METHOD_NN, 64, 64, 64, 8, 0.3, 0.2, 1.5e5)], cache_path=cache)
    with open(cache) as f:
        w, h, cap, radius, ms = (float(v) for v in f.read().split()[-5:])
    assert (w, h) in ((8, 4), (16, 2), (4, 8), (32, 1), (8, 8)) and ms > 0
    assert cap in (0, 3, 4, 5, 6) and any(abs(radius - r) < 1e-6 for r in (0.0, 0.8, 1.0, 1.2))
