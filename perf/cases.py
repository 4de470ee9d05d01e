"""What a user of the nearest-neighbour render path has it do, as cases that can be timed.

A case is a dict of plain values; ``prepare`` makes its inputs on the GPU (or on
the host, where a program holds them there), ``run`` is one pass through the
package's entry points, ``work`` what a pass cannot do without and ``exact`` the
same results from torch in 64 bits.  Clouds and G(T, n) tables have the shapes
and distributions of ``fomo_gb300.synth``: a jittered grid with a coronal loop,
and a twisted flux rope in a thin background.
"""

import math
import random
import weakref

import numpy as np
import torch

import fomo_gb300 as fg
from fomo_gb300 import synth

LINES = ((5.8, 171.073, "fe_9"), (6.0, 193.509, "fe_12"), (6.2, 211.317, "fe_14"), (6.4, 284.163, "fe_15"))
CHANNELS = (94, 131, 171, 193, 211, 335)
WIDTH = 0.6 * fg.SPEED_OF_LIGHT / 171.073  # +-0.3 Angstrom at 171, in m/s
RSUN = 695.7  # Mm


def listed():
    return [
        # the smallest call: a first look at a few points, with the neighbour indices, into host memory
        dict(name="first_look", kind="host", cloud="loop", sx=12, sy=12, sz=12, nx=16, ny=12, nz=20, L=16, l=0.3,
             b=0.2, idx=True),
        # one view at FoMoObject's default resolution, 101 x 102 pixels, 300 samples, 30 bins
        dict(name="default_resolution", kind="device", cloud="loop", sx=64, sy=61, sz=59, nx=101, ny=102, nz=300,
             L=30, l=0.4, b=-0.15),
        # the ordinary call: one 262,144-point view into a host cube
        dict(name="ordinary_view_to_host", kind="host", cloud="loop", sx=64, sy=64, sz=64, nx=128, ny=128, nz=256,
             L=64, l=0.0, b=0.0, idx=False),
        # one large spectroscopic view, left on the device for the program's next step
        dict(name="large_view", kind="device", cloud="loop", sx=128, sy=128, sz=128, nx=512, ny=512, nz=512, L=128,
             l=math.pi / 6, b=0.0),
        # a synthetic observing campaign: many views x four lines in one replayed launch
        dict(name="campaign_64_views_4_lines", kind="batch", cloud="loop", sx=128, sy=128, sz=128, views=64, lines=4,
             nx=256, ny=256, nz=512, L=64),
        # six broadband channels of one view of a clustered cloud at full resolution
        dict(name="imaging_6_channels", kind="imaging", cloud="rope", n=8388608, nx=1024, ny=1024, nz=1024, lines=6,
             l=0.6, b=0.35),
        # white light away from the equator: boxes 200 pixels wide
        dict(name="thomson_full", kind="thomson", cloud="rope", n=8388608, nx=1024, ny=1024, nz=1024, l=0.2, b=0.3),
        # the same as a quick look
        dict(name="thomson_quick_look", kind="thomson", cloud="rope", n=65536, nx=96, ny=96, nz=256, l=0.2, b=0.3),
        # the projection method, four lines of one view
        dict(name="projection_4_lines", kind="projection", cloud="loop", sx=128, sy=128, sz=128, nx=256, ny=256,
             nz=300, L=64, lines=4, l=0.5, b=0.25),
        # a simulation on the same GPU hands over each output step: index, emissivity, two lines, and on
        dict(name="simulation_step", kind="step", cloud="loop", sx=115, sy=113, sz=111, nx=256, ny=256, nz=256, L=64,
             lines=2, views=1),
        # snapshots that come from files: host arrays in, four lines of two views out to host arrays
        dict(name="host_snapshot_to_host_cubes", kind="ingest", cloud="loop", sx=128, sy=128, sz=128, nx=256, ny=256,
             nz=256, L=64, lines=4, views=2),
        # requests of mixed sizes from several users, through the server
        dict(name="served_mix", kind="serve", cloud="rope", n=4194304, requests=24, mix=5),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["host", "device", "device", "batch", "imaging", "thomson", "projection", "step", "ingest",
                       "serve"])
    view = dict(l=round(rng.uniform(0.0, math.pi / 2), 4), b=round(rng.uniform(-math.pi / 9, math.pi / 9), 4))
    side = dict(cloud="loop", sx=_log(rng, 12, 128), sy=_log(rng, 12, 128), sz=_log(rng, 12, 128))
    rope = dict(cloud="rope", n=_log(rng, 32768, 8388608))
    if kind == "host":
        return dict(kind=kind, **side, nx=_log(rng, 16, 256), ny=_log(rng, 12, 256), nz=_log(rng, 20, 512),
                    L=_log(rng, 1, 128), idx=rng.random() < 0.25, **view)
    if kind == "device":
        cloud = side if rng.random() < 0.7 else rope
        return dict(kind=kind, **cloud, nx=_log(rng, 16, 512), ny=_log(rng, 16, 512), nz=_log(rng, 20, 512),
                    L=_log(rng, 2, 128), **view)
    if kind == "batch":
        return dict(kind=kind, **side, views=_log(rng, 2, 64), lines=rng.randint(1, 4), nx=_log(rng, 32, 256),
                    ny=_log(rng, 32, 256), nz=_log(rng, 64, 512), L=_log(rng, 8, 64))
    if kind == "imaging":
        return dict(kind=kind, **rope, nx=_log(rng, 64, 1024), ny=_log(rng, 64, 1024), nz=_log(rng, 64, 1024),
                    lines=rng.randint(1, 6), **view)
    if kind == "thomson":
        return dict(kind=kind, **rope, nx=_log(rng, 64, 800), ny=_log(rng, 64, 800), nz=_log(rng, 64, 800),
                    l=view["l"], b=round(rng.uniform(0.0, 0.3), 4))
    if kind == "projection":
        return dict(kind=kind, **side, nx=_log(rng, 32, 512), ny=_log(rng, 32, 512), nz=_log(rng, 20, 512),
                    L=_log(rng, 1, 128), lines=rng.randint(1, 4), **view)
    if kind in ("step", "ingest"):
        return dict(kind=kind, **side, nx=_log(rng, 32, 256), ny=_log(rng, 32, 256), nz=_log(rng, 64, 512),
                    L=_log(rng, 2, 100), lines=rng.randint(1, 4), views=rng.randint(1, 4))
    return dict(kind="serve", cloud="rope", n=_log(rng, 262144, 4194304), requests=rng.randint(4, 24),
                mix=rng.randrange(1 << 20))


# ---------------------------------------------------------------- inputs


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _uniform(g, n, lo, hi):
    return torch.rand(n, generator=g, device="cuda", dtype=torch.float64) * (hi - lo) + lo


def _loop(sx, sy, sz, seed, centre_x=0.0):
    """x, y, z, n, T, vx, vy, vz of a coronal loop on a jittered sx x sy x sz grid over 10 Mm (float32, device)."""
    g = _gen(seed)
    ax = [torch.linspace(-5.0, 5.0, s, device="cuda", dtype=torch.float64) for s in (sx, sy, sz)]
    zz, yy, xx = torch.meshgrid(ax[2], ax[1], ax[0], indexing="ij")
    p = [v.reshape(-1) + _uniform(g, v.numel(), -0.1, 0.1) * 10.0 / (s - 1)
         for v, s in ((xx, sx), (yy, sy), (zz, sz))]
    f = 0.5 * (1.0 - torch.tanh((torch.hypot(p[0], p[1]) - 1.0) / 0.2))
    vx = 1e4 * torch.sin(2.0 * math.pi * p[2] / 10.0)
    zero = torch.zeros_like(vx)
    return [v.float().contiguous() for v in (p[0] + centre_x, p[1], p[2], f * 1e9 + (1 - f) * 1e8,
                                             f * 1e6 + (1 - f) * 2e6, vx, zero, zero)]


def _rope(n, seed, centre_x=0.0):
    """The same of a flux rope: 80 % of the points in a twisted cylinder, 20 % over the cube of 20 Mm."""
    g = _gen(seed)
    nr = int(round(0.8 * n))
    rad = 1.5 * torch.sqrt(_uniform(g, nr, 0.0, 1.0))
    zr = _uniform(g, nr, -10.0, 10.0)
    phi = _uniform(g, nr, 0.0, 2.0 * math.pi) + 2.0 * math.pi * zr / 20.0
    bg = [_uniform(g, n - nr, -10.0, 10.0) for _ in range(3)]
    perm = torch.randperm(n, generator=g, device="cuda")
    x, y, z = (torch.cat([a, b])[perm] for a, b in ((rad * torch.cos(phi), bg[0]), (rad * torch.sin(phi), bg[1]),
                                                    (zr, bg[2])))
    ne = 10.0 ** _uniform(g, n, 8.0, 10.0)
    T = 10.0 ** _uniform(g, n, math.log10(5e5), math.log10(5e6))
    rr = torch.hypot(x, y)
    v = torch.where(rr < 1.5, 1e4, 0.0) / rr.clamp(min=1e-6)
    return [a.float().contiguous() for a in (x + centre_x, y, z, ne, T, -v * y, v * x, torch.zeros_like(x))]


def _cloud(case, seed):
    cx = 1.5 * RSUN if case["kind"] == "thomson" else 0.0
    if case["cloud"] == "rope":
        return _rope(case["n"], seed, cx)
    return _loop(case["sx"], case["sy"], case["sz"], seed, cx)


def _points(case):
    return case["n"] if case["cloud"] == "rope" else case["sx"] * case["sy"] * case["sz"]


_keep = {}


def _context():
    if "ctx" not in _keep:
        _keep["ctx"] = fg.Context(0)
        _keep["stream"] = torch.cuda.Stream()
    return _keep["ctx"]


def _server():
    if "srv" not in _keep:
        _keep["srv"] = fg.Server(0)
    return _keep["srv"]


def _line_tables():
    return [synth.line_table(peak_logT=p, lambda0=lam, ion=ion) for p, lam, ion in LINES]


def _band_tables():
    return [synth.broadband_table(c, peak_logT=5.8 + 0.15 * k) for k, c in enumerate(CHANNELS)]


def _table_ids(ctx, band):
    """The tables' handles, uploaded once per context as a program does."""
    key = (id(ctx), band)
    if key not in _keep:
        _keep[key] = [ctx.table(t) for t in (_band_tables() if band else _line_tables())]
    return _keep[key]


class _State:
    """What a program keeps between renders; its snapshots go when it does."""

    def __init__(self, ctx):
        self.ctx = ctx

    def own(self, sid):
        weakref.finalize(self, self.ctx.drop_snapshot, sid).atexit = False
        return sid


def _resident(case, seed, ctx):
    torch.cuda.synchronize()
    arrays = _cloud(case, seed)
    torch.cuda.synchronize()
    return ctx.snapshot_device(arrays[0].numel(), [a.data_ptr() for a in arrays])


def _angles(case, seed):
    """(l, b) of each view: the case's own, or spread over a campaign's range."""
    if "l" in case:
        return [(case["l"], case["b"])]
    r = random.Random(seed)
    return [(r.uniform(0.0, math.pi / 2), r.uniform(-math.pi / 9, math.pi / 9)) for _ in range(case["views"])]


def _requests(case, seed, ctx, sid):
    kind = case["kind"]
    band = kind == "imaging" or case.get("L") == 1
    if kind == "thomson":
        return [ctx.request(sid, 0, fg.METHOD_THOMSON, case["nx"], case["ny"], case["nz"], 1, l, b)
                for l, b in _angles(case, seed)]
    tids = _table_ids(ctx, band)[: case.get("lines", 1)]
    method = fg.METHOD_PROJECTION if kind == "projection" else fg.METHOD_NN
    return [ctx.request(sid, t, method, case["nx"], case["ny"], case["nz"], 1 if band else case["L"], l, b, WIDTH)
            for l, b in _angles(case, seed) for t in tids]


def _serve_mix(case, seed, ctx, sids):
    """Sizes from the case, views from the seed."""
    r, v = random.Random(case["mix"]), random.Random(seed)
    lines, bands = _table_ids(ctx, False), _table_ids(ctx, True)
    reqs = []
    while len(reqs) < case["requests"]:
        px, L = r.choice([64, 100, 128, 200, 256, 512, 700]), r.choice([1, 1, 16, 30, 64, 128])
        if px * px * L > 1 << 22:
            continue
        t = r.choice(bands if L == 1 else lines)
        reqs.append(ctx.request(r.choice(sids), t, fg.METHOD_NN, px, px, 256, L, v.uniform(0.0, math.pi / 2),
                                v.uniform(-math.pi / 9, math.pi / 9), WIDTH))
    return reqs


def prepare(case, seed):
    kind = case["kind"]
    if kind == "serve":
        srv = _server()
        s = _State(srv.ctx)
        s.kind, s.srv = kind, srv
        sids = []
        for k, part in enumerate((8, 3, 2, 1)):  # several snapshots of different sizes, as a server holds them
            c = dict(case, n=max(1024, case["n"] // part))
            sids.append(s.own(_resident(c, seed * 4 + k, srv.ctx)))
        s.reqs = _serve_mix(case, seed, srv.ctx, sids)
        s.outs = [np.empty(fg.Context.cube_shape(q), np.float32) for q in s.reqs]
        return s
    ctx = _context()
    s = _State(ctx)
    s.kind, s.case, s.seed = kind, case, seed
    if kind in ("step", "ingest"):
        arrays = _cloud(case, seed)
        torch.cuda.synchronize()
        s.arrays = arrays if kind == "step" else synth.Snapshot(*[a.cpu().numpy() for a in arrays])
    else:
        s.reqs = _requests(case, seed, ctx, s.own(_resident(case, seed, ctx)))
    nv, nl = case.get("views", 1), case.get("lines", 1)
    band = kind in ("imaging", "thomson") or case.get("L") == 1
    shape = (nv, nl, case["ny"], case["nx"], 1 if band else case["L"])
    if kind == "ingest":
        s.out = np.zeros(shape, np.float32)
    elif kind != "host":
        s.out = torch.empty(shape, dtype=torch.float32, device="cuda")
        size = s.out[0, 0].numel() * 4
        s.ptrs = [s.out.data_ptr() + k * size for k in range(nv * nl)]
        torch.cuda.synchronize()
    return s


def run(s):
    ctx, kind = s.ctx, s.kind
    if kind == "serve":
        tickets = [s.srv.submit(q, o) for q, o in zip(s.reqs, s.outs)]
        for t in tickets:
            s.srv.wait(t)
        return s.outs
    if kind == "host":
        cube, idx, info = ctx.render(s.reqs[0], want_idx=s.case["idx"])
        view = np.array([info.minx, info.maxx, info.miny, info.maxy, info.maxdistance, info.pathlength])
        return {"cube": cube, "view": view, **({"idx": idx} if s.case["idx"] else {})}
    if kind in ("step", "ingest"):
        if kind == "step":
            sid = ctx.snapshot_device(s.arrays[0].numel(), [a.data_ptr() for a in s.arrays])
        else:
            sid = ctx.snapshot(s.arrays)
        reqs = _requests(s.case, s.seed, ctx, sid)
        if kind == "step":
            ctx.render_batch_device(reqs, s.ptrs)
        else:
            ctx.render_batch(reqs, outs=list(s.out.reshape(len(reqs), *s.out.shape[2:])))
        ctx.drop_snapshot(sid)
        return s.out
    stream = _keep["stream"].cuda_stream
    if len(s.reqs) == 1:
        ctx.render_device(s.reqs[0], s.ptrs[0], stream=stream)
    else:
        ctx.render_batch_device(s.reqs, s.ptrs, stream=stream, graph=kind == "batch")
    return s.out


def _mix_sizes(case):
    """(points, requests) of a server's mix without its handles."""
    r = random.Random(case["mix"])
    got = []
    while len(got) < case["requests"]:
        px, L = r.choice([64, 100, 128, 200, 256, 512, 700]), r.choice([1, 1, 16, 30, 64, 128])
        if px * px * L > 1 << 22:
            continue
        r.choice(range(6 if L == 1 else 4))
        r.choice(range(4))
        got.append((px, L))
    return got


def work(case):
    """Each array of the points read once, each cube written once; per line-of-sight sample its position (6) and the
    distance to its neighbour (8), per sample and line one addition and product."""
    if case["kind"] == "serve":
        n = sum(max(1024, case["n"] // part) for part in (8, 3, 2, 1))
        mix = _mix_sizes(case)
        return {"bytes": n * 32 + sum(4 * px * px * L for px, L in mix), "flops": sum(px * px * 256 * 16 for px, _ in mix)}
    n, nv, nl = _points(case), case.get("views", 1), case.get("lines", 1)
    L = 1 if case["kind"] in ("imaging", "thomson") else case["L"]
    rays = case["nx"] * case["ny"] * nv
    out = 4 * rays * nl * L + (4 * rays * case["nz"] if case.get("idx") else 0)
    if case["kind"] == "projection":
        return {"bytes": n * 32 + out, "flops": n * (20 + 6 * nl * L)}
    return {"bytes": n * 32 + out, "flops": rays * case["nz"] * (14 + 2 * nl)}


# ---------------------------------------------------------------- the same in 64 bits


def _emission64(arrays, t, imaging):
    """eps and width of every point: n^2 G(T, n) / w, G linear in log T and nearest in log n."""
    ne, T = arrays[3].double(), arrays[4].double()
    logT = torch.from_numpy(t.logT).cuda().double()
    G = torch.from_numpy(t.G).cuda().double()
    step = float(logT[1] - logT[0])
    lT, ln = torch.log10(T), torch.log10(ne)
    i = torch.floor((lT - logT[0]) / step).long()
    # the density row is the nearest in the table's 32-bit axis
    r32 = (ln.float() - float(t.logn[0])) / float(t.logn[1] - t.logn[0])
    j = torch.floor(r32 + 0.5).long()
    ok = (i >= 0) & (i + 1 <= t.nt - 1) & (j >= 0) & (j <= t.nrho - 1)
    i, j = i.clamp(0, t.nt - 2), j.clamp(0, t.nrho - 1)
    g = G[j, i] + (lT - logT[i]) / (logT[i + 1] - logT[i]) * (G[j, i + 1] - G[j, i])
    g = torch.where(ok, g, torch.zeros_like(g))
    if imaging:
        return ne * ne * g, torch.ones_like(g)
    w = 2 * math.sqrt(2 * math.log(2)) * math.sqrt(1.3806504e-23 / 1.67262158e-27 / t.atweight) * t.lambda0 / 2.99792458e8
    w = w * torch.sqrt(T)
    return ne * ne * g / w / 1.0645, w  # a Gaussian of that full width and unit area (the method's rounded constant)


def _rotated(arrays, l, b):
    x, y, z = (a.double() for a in arrays[:3])
    cl, sl, cb, sb = math.cos(l), math.sin(l), math.cos(b), math.sin(b)
    return x * cb * cl - y * cb * sl - z * sb, x * sl + y * cl, x * sb * cl - y * sb * sl + z * cb


def _range(v):
    return float(v.min()), float(v.max())


def _thomson_terms(arrays, l, b):
    """n times the polarised scattering term, sin^2 of the scattering angle and the blended coordinates of each point."""
    x, y, z, ne = (a.double() for a in arrays[:4])
    r = torch.sqrt(x * x + y * y + z * z)
    so = RSUN / r
    ss = so * so
    cs = 1 - ss
    co = torch.sqrt(cs)
    lt = torch.log((1 + so) / co)
    u = 0.58
    a = co * ss
    bb = -1.0 / 8 * (1 - 3 * ss - cs * (1 + 3 * ss) / so * lt)
    pol = a + u * (bb - a)
    eps = 1e-6
    cb, sb = math.cos(b), math.sin(b)
    cb = eps if abs(cb) < eps else cb
    sb = eps if abs(sb) < eps else sb
    cl, sl = math.cos(l), math.sin(l)
    blend = 1.0 / (1.0 + math.exp(-20.0 * (abs(b) - 1.309)))
    p = [x * cb * cl - y * cb * sl - z * sb, x * sl + y * cl, x * sb * cl - y * sb * sl + z * cb]
    q = [x * cl - y * sl, x * sl + y * cl, z]
    p = [(1 - blend) * i + blend * j for i, j in zip(p, q)]
    ip = sb * cl * p[0] - sb * sl * p[1] + cb * p[2]
    s2 = 1 - ip * ip / (p[0] * p[0] + p[1] * p[1] + p[2] * p[2])
    return ne * pol, s2, p


def _lambda64(t, L):
    lw = WIDTH * t.lambda0 / fg.SPEED_OF_LIGHT
    return torch.arange(L, device="cuda", dtype=torch.float64) / max(L - 1, 1) * lw - lw / 2


def _spectra64(eps, w, v, lam, t, idx):
    """Line profiles of the points idx (-1: none) summed over the last axis: [..., L]."""
    e = torch.where(idx >= 0, eps[idx.clamp(min=0)], torch.zeros((), device="cuda", dtype=torch.float64))
    iw = 1.0 / w[idx.clamp(min=0)]
    shift = v[idx.clamp(min=0)] * (t.lambda0 / fg.SPEED_OF_LIGHT)
    out = torch.empty(*idx.shape[:-1], lam.numel(), device="cuda", dtype=torch.float64)
    for m in range(lam.numel()):
        out[..., m] = (e * torch.exp(-4 * math.log(2) * ((lam[m] - shift) * iw) ** 2)).sum(-1)
    return out


def _neighbours64(arrays, l, b, px, py, pz, md, pairs):
    """Index of the nearest point strictly inside the box around each sample (32-bit targets and box corners, as the
    method defines them), -1 where it holds none: [ny, nx, nz]; None when it would take more than `pairs` distances."""
    cl, sl, cb, sb = math.cos(l), math.sin(l), math.cos(b), math.sin(b)
    pts = torch.stack([a.double() for a in arrays[:3]], 1)
    rot = torch.stack(_rotated(arrays, l, b), 1)
    reach = math.sqrt(3.0) * md * 1.0001 + 1e-3
    ny, nx, nz = py.numel(), px.numel(), pz.numel()
    idx = torch.full((ny, nx, nz), -1, dtype=torch.int64, device="cuda")
    spent = 0
    tile, zt = 8, 64
    for i0 in range(0, ny, tile):
        yy = py[i0:i0 + tile]
        strip = ((rot[:, 1] > yy.min() - reach) & (rot[:, 1] < yy.max() + reach)).nonzero()[:, 0]
        for j0 in range(0, nx, tile):
            xx = px[j0:j0 + tile]
            r0 = rot[strip, 0]
            col = strip[(r0 > xx.min() - reach) & (r0 < xx.max() + reach)]
            if col.numel() == 0:
                continue
            rz = rot[col, 2]
            for k0 in range(0, nz, zt):
                zz = pz[k0:k0 + zt]
                near = col[(rz > zz.min() - reach) & (rz < zz.max() + reach)]
                if near.numel() == 0:
                    continue
                gy, gx, gz = torch.meshgrid(yy, xx, zz, indexing="ij")
                p = torch.stack([gx * cb * cl + gy * sl + gz * sb * cl, -gx * cb * sl + gy * cl - gz * sb * sl,
                                 -gx * sb + gz * cb], -1).reshape(-1, 3)
                spent += p.shape[0] * near.numel()
                if spent > pairs:
                    return None
                best = torch.full((p.shape[0],), math.inf, device="cuda", dtype=torch.float64)
                at = torch.full((p.shape[0],), -1, device="cuda", dtype=torch.int64)
                t, lo, hi = p.float().double(), (p - md).float().double(), (p + md).float().double()
                for c0 in range(0, near.numel(), 8192):
                    c = near[c0:c0 + 8192]
                    d = torch.zeros(p.shape[0], c.numel(), device="cuda", dtype=torch.float64)
                    for k in range(3):
                        q = pts[c, k][None, :]
                        d += (q - t[:, k, None]) ** 2
                        d.masked_fill_((q <= lo[:, k, None]) | (q >= hi[:, k, None]), math.inf)
                    v, a = d.min(1)
                    take = v < best
                    best, at = torch.where(take, v, best), torch.where(take, c[a], at)
                idx[i0:i0 + tile, j0:j0 + tile, k0:k0 + zt] = at.reshape(gx.shape)
    return idx


def _geometry(case, l, b, p):
    """Ray positions, LOS positions, box half-width and path length of a view whose rotated points are p."""
    (x0, x1), (y0, y1), (z0, z1) = (_range(v) for v in p)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    f64 = dict(device="cuda", dtype=torch.float64)
    px = torch.arange(nx, **f64) / (nx - 1) * (x1 - x0) + x0
    py = torch.arange(ny, **f64) / (ny - 1) * (y1 - y0) + y0
    dz = (z1 - z0) / (nz - 1) if nz > 1 else z1 - z0
    pz = torch.arange(nz, **f64) * dz + z0
    sx, sy = (x1 - x0) / (nx - 1), (y1 - y0) / (ny - 1)
    if case["kind"] == "thomson":
        mix = 1.0 / (1.0 + math.exp(-10 * (abs(b) - 0.1745)))
        equator = max(0.5 * math.hypot(sx, sy), 0.1 * sx)
        md = equator * (1 - mix) + max(sx, sy) / 0.005 * mix
    else:
        md = max(sx, sy) / 0.3
    return px, py, pz, md, dz if nz > 1 and z1 != z0 else 1.0, (x0, x1, y0, y1)


def exact(case, seed):
    kind = case["kind"]
    n = _points(case)
    # pairs a search may test within about ten seconds
    most = 1.6e11
    if kind == "serve" or case["nx"] * case["ny"] * case["nz"] * case.get("views", 1) > 1.5e8:
        return None
    arrays = _cloud(case, seed)
    tables = (_band_tables() if kind == "imaging" or case.get("L") == 1 else _line_tables())[: case.get("lines", 1)]
    spectral = kind != "thomson" and kind != "imaging" and case["L"] > 1
    views = _angles(case, seed)
    if kind != "projection" and len(views) * case["nx"] * case["ny"] * case["nz"] * len(tables) * case.get("L", 1) > 4e10:
        return None
    out = []
    view = idx = None
    for l, b in views:
        if kind == "thomson":
            pol, s2, p = _thomson_terms(arrays, l, b)
        else:
            p = _rotated(arrays, l, b)
        px, py, pz, md, path, ext = _geometry(case, l, b, p)
        view = np.array([*ext, md, path])
        dn = 1.0
        if kind != "thomson" and tables[0].is_dn:
            # the solid angle of a pixel: its sides in arcseconds at 1 AU
            dn = (ext[1] - ext[0]) / (case["nx"] - 1) / 0.715 * (ext[3] - ext[2]) / (case["ny"] - 1) / 0.715
            dn *= (math.pi / 180 / 3600) ** 2
        scale = path * 1e8 * dn
        v = math.sin(b) * math.cos(l) * arrays[5].double() - math.sin(b) * math.sin(l) * arrays[6].double() + \
            math.cos(b) * arrays[7].double()
        if kind == "projection":
            j = torch.floor((p[0] - ext[0]) / (ext[1] - ext[0]) * (case["nx"] - 1) + 0.5).long()
            i = torch.floor((p[1] - ext[2]) / (ext[3] - ext[2]) * (case["ny"] - 1) + 0.5).long()
            pix = i * case["nx"] + j
            for t in tables:
                eps, w = _emission64(arrays, t, not spectral)
                L = case["L"]
                cube = torch.zeros(case["ny"] * case["nx"], L, device="cuda", dtype=torch.float64)
                lam = _lambda64(t, L)
                for m in range(L):
                    add = eps
                    if spectral:
                        add = eps * torch.exp(-4 * math.log(2) * ((lam[m] - v * (t.lambda0 / fg.SPEED_OF_LIGHT)) / w) ** 2)
                    cube[:, m].index_add_(0, pix, add)
                out.append((cube * scale).reshape(case["ny"], case["nx"], L).cpu())
            continue
        idx = _neighbours64(arrays, l, b, px, py, pz, md, most / len(views))
        if idx is None:
            return None
        if kind == "thomson":
            const = 0.5 * math.pi * 2.8179e-13 ** 2 * 2.8e10 / (1 - 0.58 / 3)
            pb = (pol * s2).clamp(min=0)
            val = torch.where(idx >= 0, pb[idx.clamp(min=0)], torch.zeros((), device="cuda", dtype=torch.float64))
            out.append((val.sum(-1, keepdim=True) * const * scale).cpu())
            continue
        for t in tables:
            eps, w = _emission64(arrays, t, not spectral)
            if spectral:
                rows = [_spectra64(eps, w, v, _lambda64(t, case["L"]), t, idx[i:i + 16]) for i in range(0, case["ny"], 16)]
                out.append((torch.cat(rows) * scale).cpu())
            else:
                e = torch.where(idx >= 0, eps[idx.clamp(min=0)], torch.zeros((), device="cuda", dtype=torch.float64))
                out.append((e.sum(-1, keepdim=True) * scale).cpu())
    cube = torch.stack(out).reshape(len(views), -1, *out[0].shape)
    if kind == "host":
        return {"cube": cube[0, 0], "view": view, **({"idx": idx} if case["idx"] else {})}
    return cube
