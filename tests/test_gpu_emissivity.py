"""Per-point emissivity against its FP64 expression, bit for bit.

Every FP64 intermediate (log10, 10^x, the table's interpolation, the two scalings)
is rounded to FP32 at once, and the kernel gets that rounding from pairs of FP32
numbers where it can.  numpy evaluates the same expressions in FP64.  The device's
and the host's FP64 log10 and pow may differ by an ulp of FP64, which changes the
rounding to FP32 of about one value in 2^28: at most one value in a million may
differ, by at most one FP32 ulp of eps per factor (four).
"""

import numpy as np
import pytest

import fomo_gb300 as fg
from fomo_gb300 import synth

pytestmark = pytest.mark.gpu


def _expected(n, T, t, imaging, abund):
    with np.errstate(all="ignore"):
        f32, f64 = np.float32, np.float64
        logn = np.where(n <= 0, f32(0), np.log10(n.astype(f64)).astype(f32))
        lT = np.where(T <= 0, f32(0), np.log10(T.astype(f64)).astype(f32))
        qT = np.floor((lT - t.logT[0]) / (t.logT[1] - t.logT[0]))
        q = (logn - t.logn[0]) / (t.logn[1] - t.logn[0])
        qR = np.where(q - np.floor(q) >= 0.5, np.floor(q) + 1, np.floor(q))
        ok = (qT >= 0) & (qT + 1 <= t.nt - 1) & (qR >= 0) & (qR <= t.nrho - 1)
        i, j = np.where(ok, qT, 0).astype(int), np.where(ok, qR, 0).astype(int)
        x1, y1 = t.logT[i + 1].astype(f64), t.G[j, i + 1].astype(f64)
        x2, y2 = t.logT[i].astype(f64), t.G[j, i].astype(f64)
        g = np.where(ok, ((lT.astype(f64) - x1) * (y2 - y1) / (x2 - x1) + y1).astype(f32), f32(0))
        if imaging:
            w, k = np.ones_like(g), 1.0
        else:
            cw = 2 * np.sqrt(2 * np.log(2)) * np.sqrt(1.3806504e-23 / 1.67262158e-27 / t.atweight) * t.lambda0 / 2.99792458e8
            w = (cw * np.sqrt(T).astype(f64)).astype(f32)
            k = 1.0 / 1.0645 * abund
        b = np.power(10.0, (2.0 * logn.astype(f64)).astype(f32).astype(f64)).astype(f32)
        d = (k * (b * g).astype(f64)).astype(f32)
        return (d / w).astype(f32), w.astype(f32)


@pytest.mark.parametrize("imaging", [False, True])
@pytest.mark.parametrize("values", ["corona", "wide", "edges"])
def test_bits(values, imaging):
    rng = np.random.default_rng(7)
    m = 400_000
    if values == "corona":
        n, T = 10.0 ** rng.uniform(7.5, 12.5, m), 10.0 ** rng.uniform(3.8, 8.2, m)
    elif values == "wide":
        n, T = 10.0 ** rng.uniform(-37, 38, m), 10.0 ** rng.uniform(-37, 38, m)
    else:  # powers of two and ten, table nodes, zeros, negatives, the smallest and largest numbers
        special = np.concatenate([2.0 ** np.arange(-149, 128), 10.0 ** np.arange(-38, 39.0), [0.0, -1.0, -1e9, 1e-45, 3.4e38],
                                  10.0 ** np.linspace(4, 8, 101), 10.0 ** np.linspace(8, 12, 41)])
        n, T = rng.choice(special, m), np.abs(rng.choice(special, m))
    s = synth.loop_snapshot(8, seed=1)
    pos = rng.uniform(-5, 5, (3, m))
    s = synth.Snapshot(*[np.asarray(a, np.float32) for a in (*pos, n, T, np.zeros(m), np.zeros(m), np.zeros(m))])
    t = synth.broadband_table(171) if imaging else synth.line_table()
    with fg.Context(0) as ctx:
        eps, w = ctx.emission(ctx.snapshot(s), ctx.table(t), imaging=imaging, abundratio=1.0 if imaging else 0.7)
    want_e, want_w = _expected(s.n, s.T, t, imaging, 0.7)
    np.testing.assert_array_equal(w, want_w)
    off = ~((eps == want_e) | (np.isnan(eps) & np.isnan(want_e)))
    assert off.mean() <= 1e-6, (off.sum(), eps[off][:5], want_e[off][:5])
    assert (np.abs(eps[off] - want_e[off]) <= 4 * np.spacing(np.abs(want_e[off]))).all()
