"""The work that programs give this engine, as measurable cases.

Every case goes through the public Python binding (``terranni_b200.engine``),
the way a program calls it, over seeded synthetic LiDAR clouds made on the
device: 70 % uniform and 30 % clustered points, empty circular lakes, an
eight-octave relief, int32 LAS units of 0.01 m.

Kinds of case
  call        one work package through ``Engine.interpolate_device``: point
              rows and the output grid in device memory, queued, no statistics
              (what ``nni::performNNI`` is called for, tile by tile)
  batch       many uneven work packages as one planned, graph-captured launch
              sequence (``Engine.batch``), on device buffers or (host) from and
              to pinned host memory
  segment     one large grid from host points in tiles with halos
              (``Engine.segment_run``)
  served      requests against a resident cloud, all submitted at once and
              waited for (``Engine.server``)
  spacetime   one work package at one time with a time radius
              (``Engine.interpolate_spacetime_device``)
  compat      one work package with the reference's own default semantics
              (``Engine.interpolate_compat_device``)
"""
import math

import numpy as np
import torch

from terranni_b200 import engine, synth

DEV = "cuda"
_engine = None


def the_engine():
    """One context for the whole program, as a program keeps it."""
    global _engine
    if _engine is None:
        _engine = engine.Engine(device=0)
    return _engine


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------

def call(ncols, nrows, cell, points, lakes=0, halo=0, site=False, gid=False):
    return {"kind": "call", "ncols": ncols, "nrows": nrows, "cell": cell, "points": points, "lakes": lakes,
            "halo": halo, "site": site, "gid": gid}


def batch(tiles, lo, hi, layout, host=False, small_radius=0, bin_target=0):
    return {"kind": "batch", "tiles": tiles, "lo": lo, "hi": hi, "layout": layout, "host": host,
            "small_radius": small_radius, "bin_target": bin_target}


def segment(ncols, nrows, cell, points, lakes):
    return {"kind": "segment", "ncols": ncols, "nrows": nrows, "cell": cell, "points": points, "lakes": lakes}


def served(side_m, points, lakes, requests, most_m, layout):
    return {"kind": "served", "side_m": side_m, "points": points, "lakes": lakes, "requests": requests,
            "most_m": most_m, "layout": layout}


def spacetime(ncols, nrows, cell, points, lakes, radius):
    return {"kind": "spacetime", "ncols": ncols, "nrows": nrows, "cell": cell, "points": points, "lakes": lakes,
            "radius": radius}


def compat(ncols, nrows, scale, points):
    return {"kind": "compat", "ncols": ncols, "nrows": nrows, "scale": scale, "points": points}


def listed():
    return [
        # the smallest work packages: an interactive preview or one small tile of a loop over many; launches and latency
        dict(call(96, 80, 100, 6000), name="call_96"),
        # the reference-path workload: 512 x 512 cells at 1 m, 200 k points, with the site map
        dict(call(512, 512, 100, 200_000, site=True), name="call_512_site"),
        # a work package as the C++ shim plans it: ragged sides, a raster halo, the stream's own point ids
        dict(call(1237, 811, 50, 1_900_003, lakes=2, halo=11, gid=True, site=True), name="call_1237_halo"),
        # thin data: a sparse airborne strip with lakes, most discs many cells wide
        dict(call(1500, 1400, 100, 170_000, lakes=4), name="call_1500_sparse"),
        # a whole survey tile: 4096 x 4096 cells at 1 m, 20 M points, lakes
        dict(call(4096, 4096, 100, 20_000_000, lakes=16), name="call_4096"),
        # a production batch of uneven tiles (sides 64 to 1024 cells, 0.05 to 8 points per cell), engine defaults
        dict(batch(1024, 64, 1024, 1), name="batch_1024"),
        # the same mix in a smaller batch with the options that the autotuner settles on
        dict(batch(200, 64, 1024, 2, small_radius=2, bin_target=2), name="batch_200_tuned"),
        # the same mix end to end, from pinned host points to pinned host heights
        dict(batch(200, 64, 1024, 3, host=True), name="batch_200_host"),
        # one large grid streamed from host memory in tiles with halos
        dict(segment(5000, 4200, 100, 24_000_000, 20), name="segment_5000"),
        # a burst of requests of uneven size against a resident cloud
        dict(served(5000.0, 12_000_000, 24, 24, 2048.0, 4), name="served_24"),
        # space-time: five slices of a time series at one time step
        dict(spacetime(1536, 1200, 100, 4_000_000, 4, 2), name="spacetime_1536"),
        # the reference's own default semantics at its default scale of 5 pixels per cell
        dict(compat(1000, 900, 5, 3_600_000), name="compat_1000"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    cell = rng.choice([50, 100, 200])
    k = rng.random()
    if k < 0.45:
        nc, nr = _log(rng, 64, 4096), _log(rng, 64, 4096)
        n = min(20_000_000, max(1000, int(nc * nr * math.exp(rng.uniform(math.log(0.05), math.log(8.0))))))
        return call(nc, nr, cell, n, rng.randrange(0, 9), rng.choice([0, 0, 3, 17, 40]), rng.random() < 0.4,
                    rng.random() < 0.3)
    if k < 0.70:
        lo = _log(rng, 64, 256)
        hi = min(1024, lo * rng.choice([2, 4, 8]))
        most = 1.2e8 / ((hi * hi - lo * lo) / (2.0 * math.log(hi / lo)))    # 120 M cells: fewer than the largest listed
        return batch(_log(rng, 8, min(800, most)), lo, hi, rng.randrange(100, 1 << 30),
                     rng.random() < 0.25, rng.choice([0, 0, 1, 2, 4]), rng.choice([0, 0, 1, 2, 6]))
    if k < 0.78:
        nc, nr = _log(rng, 1500, 5000), _log(rng, 1500, 4200)
        return segment(nc, nr, cell, int(nc * nr * rng.uniform(0.3, 1.1)), rng.randrange(0, 20))
    if k < 0.84:
        side = rng.uniform(2500.0, 5000.0)
        return served(side, int(side * side * 0.48), rng.randrange(0, 24), _log(rng, 4, 32), rng.uniform(512.0, 2048.0),
                      rng.randrange(100, 1 << 30))
    if k < 0.92:
        nc, nr, rt = _log(rng, 128, 1536), _log(rng, 128, 1200), rng.choice([0, 1, 2, 3])
        return spacetime(nc, nr, cell, max(2000, int(nc * nr * rng.uniform(0.3, 2.2))), rng.randrange(0, 5), rt)
    nc, nr = _log(rng, 100, 1000), _log(rng, 100, 900)
    return compat(nc, nr, rng.choice([1, 2, 5]), max(500, int(4 * nc * nr * rng.uniform(0.2, 1.0))))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) * 7919 + 13)
    return g


def _terrain(gen, counts, ext, lakes, rmin, rmax, clusters=8):
    """Clouds of several tiles at once: counts points per tile, each in its
    ext (w, h) box of LAS units at the origin, with `lakes` empty discs of
    radius rmin..rmax times the shorter side -> int32 (sum, 3) on the device."""
    T = len(counts)
    cnt = torch.tensor(counts, device=DEV)
    ext = torch.tensor(ext, dtype=torch.float64, device=DEV)
    n = int(sum(counts))
    short = ext.min(1).values
    tid = torch.repeat_interleave(torch.arange(T, device=DEV), cnt, output_size=n)

    def rnd(*shape):
        return torch.rand(*shape, generator=gen, device=DEV, dtype=torch.float64)

    cc = rnd(T, clusters, 2) * ext[:, None, :]
    sigma = (short / 50.0).clamp(min=100.0)
    L = max(max(lakes), 1)
    lc = rnd(T, L, 2) * ext[:, None, :]
    lr = (rmin + (rmax - rmin) * rnd(T, L)) * short[:, None]
    lr[torch.arange(L, device=DEV)[None, :] >= torch.tensor(lakes, device=DEV)[:, None]] = -1.0
    e = ext[tid]
    xy = rnd(n, 2) * e
    pick = rnd(n) < 0.3
    which = torch.randint(0, clusters, (n,), generator=gen, device=DEV)
    blob = cc[tid, which] + torch.randn(n, 2, generator=gen, device=DEV, dtype=torch.float64) * sigma[tid][:, None]
    fits = ((blob >= 0) & (blob < e)).all(1)
    xy = torch.where((pick & fits)[:, None], blob, xy)
    del blob, pick, which, fits
    if max(lakes) > 0:
        # points that fall in a lake are drawn again, uniformly, and the few
        # left after three rounds are pushed out to the shore
        for k in range(4):
            wet = torch.zeros(n, dtype=torch.bool, device=DEV)
            for j in range(L):
                d = xy - lc[tid, j]
                r = lr[tid, j]
                inside = (r > 0) & ((d * d).sum(1) < r * r)
                if k == 3:
                    d = d + 1e-3
                    xy = torch.where(inside[:, None], lc[tid, j] + d * (r / (d * d).sum(1).sqrt())[:, None], xy)
                else:
                    wet |= inside
            if k < 3:
                xy = torch.where(wet[:, None], rnd(n, 2) * e, xy)
    xy = xy.floor().clamp(min=0)
    xy = torch.minimum(xy, e - 1)
    z = torch.full((n,), 15000.0, device=DEV, dtype=torch.float64)
    fx, fy, ph = rnd(8), rnd(8), rnd(8)
    for k in range(8):
        u = xy / (short[tid][:, None] / 2.0) * (2.0 ** k * 2.0 * math.pi)
        z += 6000.0 * 2.0 ** (-0.8 * k) * torch.sin(u[:, 0] * (0.5 + fx[k]) + u[:, 1] * (0.5 - fy[k]) + 6.3 * ph[k])
    z += 10.0 * torch.randn(n, generator=gen, device=DEV, dtype=torch.float64)
    return torch.cat([xy, z.floor()[:, None]], 1).to(torch.int32)


def _cloud(case, seed, w, h, rmin, rmax, clusters=64):
    return _terrain(_gen(seed), [case["points"]], [(w, h)], [case["lakes"]], rmin, rmax, clusters)


def _specs(case):
    """Tiles of a batch: side log-uniform in [lo, hi] cells, cell 0.5/1/2 m,
    0.05 to 8 points per cell (at least 1000 points, at most 1 M), 0 to 4 lakes."""
    r = np.random.default_rng(case["layout"])
    T = case["tiles"]
    side = np.exp(r.uniform(math.log(case["lo"]), math.log(case["hi"]), T)).astype(np.int64)
    cell = r.choice(np.array([50, 100, 200]), T)
    dens = np.exp(r.uniform(math.log(0.05), math.log(8.0), T))
    n = np.clip((dens * side * side).astype(np.int64), 1000, 1_000_000)
    lakes = r.integers(0, 5, T)
    return [(int(side[k]), int(cell[k]), int(n[k]), int(lakes[k])) for k in range(T)]


def _requests(case):
    r = np.random.default_rng(case["layout"])
    out = []
    for _ in range(case["requests"]):
        side = math.exp(r.uniform(math.log(128.0), math.log(case["most_m"])))
        cell = int(r.choice(np.array([50, 100, 200])))
        k = max(1, int(round(side * 100 / cell)))
        room = max(1, int(case["side_m"] * 100) - k * cell)
        out.append((int(r.integers(0, room)), int(r.integers(0, room)), k, cell))
    return out


def _call_points(case, seed):
    h, cs = case["halo"], case["cell"]
    xyz = _cloud(case, seed, (case["ncols"] + 2 * h) * cs, (case["nrows"] + 2 * h) * cs, 0.012, 0.1)
    xyz[:, :2] -= h * cs
    return xyz


def _call_wp(case):
    h = case["halo"]
    raster = (-h, -h, case["ncols"] + h, case["nrows"] + h) if h else None
    return engine.make_wp(case["ncols"], case["nrows"], case["cell"], raster=raster)


def _call_gid(case, seed):
    return torch.randperm(case["points"], generator=_gen(seed + 1), device=DEV).to(torch.int32)


def _batch_points(case, seed):
    sp = _specs(case)
    xyz = _terrain(_gen(seed), [s[2] for s in sp], [(s[0] * s[1],) * 2 for s in sp], [s[3] for s in sp], 0.05, 0.3)
    org = torch.tensor([synth.tile_origin(k) for k in range(len(sp))], dtype=torch.int32, device=DEV)
    tid = torch.repeat_interleave(torch.arange(len(sp), device=DEV), torch.tensor([s[2] for s in sp], device=DEV),
                                  output_size=xyz.shape[0])
    xyz[:, :2] += org[tid]
    return sp, xyz, tid


def _st_times(case, seed):
    rt = case["radius"]
    return torch.randint(50 - 2 * rt, 51 + 2 * rt, (case["points"],), generator=_gen(seed + 2), device=DEV,
                         dtype=torch.int32)


def _pinned(t):
    return torch.empty(t.shape, dtype=t.dtype, pin_memory=True).copy_(t)


def prepare(case, seed):
    eng, kind = the_engine(), case["kind"]
    s = {"kind": kind}
    if kind == "call":
        h = case["halo"]
        s["wp"], s["xyz"] = _call_wp(case), _call_points(case, seed)
        s["gid"] = _call_gid(case, seed) if case["gid"] else None
        s["h"] = torch.empty(case["nrows"], case["ncols"], dtype=torch.float32, device=DEV)
        s["site"] = torch.empty(case["nrows"] + 2 * h, case["ncols"] + 2 * h, dtype=torch.int32,
                                device=DEV) if case["site"] else None
    elif kind == "batch":
        sp, xyz, tid = _batch_points(case, seed)
        idx = tid[:, None].expand(-1, 2)
        lo = torch.full((len(sp), 2), 2 ** 31 - 1, dtype=torch.int32, device=DEV).scatter_reduce(0, idx, xyz[:, :2],
                                                                                               "amin").cpu().tolist()
        hi = torch.full((len(sp), 2), -2 ** 31, dtype=torch.int32, device=DEV).scatter_reduce(0, idx, xyz[:, :2],
                                                                                            "amax").cpu().tolist()
        tiles, pt, out = [], 0, 0
        for k, (side, cell, n, _) in enumerate(sp):
            ox, oy = synth.tile_origin(k)
            tiles.append(engine.make_tile(engine.make_wp(side, side, cell, ox, oy), pt, n, out,
                                          extent=(*lo[k], *hi[k])))
            pt += n
            out += side * side
        s["batch"] = eng.batch(tiles, small_radius=case["small_radius"], bin_target=case["bin_target"], use_graph=True,
                               order_by_cost=True)
        s["host"] = case["host"]
        if case["host"]:
            s["keep"] = (_pinned(xyz), torch.empty(out, dtype=torch.float32, pin_memory=True))
            s["xyz"], s["h"] = (t.numpy() for t in s["keep"])
        else:
            s["xyz"], s["h"] = xyz, torch.empty(out, dtype=torch.float32, device=DEV)
    elif kind == "segment":
        xyz = _cloud(case, seed, case["ncols"] * case["cell"], case["nrows"] * case["cell"], 0.012, 0.08)
        s["keep"] = (_pinned(xyz), torch.empty(case["nrows"], case["ncols"], dtype=torch.float32, pin_memory=True))
        s["xyz"], s["h"] = (t.numpy() for t in s["keep"])
        s["args"] = (case["ncols"], case["nrows"], case["cell"])
    elif kind == "served":
        side = int(case["side_m"] * 100)
        xyz = _cloud(case, seed, side, side, 0.012, 0.05).cpu().numpy()
        s["server"] = eng.server(xyz, slot_bytes=2 << 30)
        s["requests"] = _requests(case)
        s["out"] = [torch.empty(k, k, dtype=torch.float32, pin_memory=True).numpy() for _, _, k, _ in s["requests"]]
    elif kind == "spacetime":
        s["wp"] = engine.make_wp(case["ncols"], case["nrows"], case["cell"])
        s["xyz"] = _cloud(case, seed, case["ncols"] * case["cell"], case["nrows"] * case["cell"], 0.03, 0.12)
        s["t"], s["radius"] = _st_times(case, seed), case["radius"]
        s["h"] = torch.empty(case["nrows"], case["ncols"], dtype=torch.float32, device=DEV)
    elif kind == "compat":
        side = (case["ncols"] * 200, case["nrows"] * 200)
        s["xyz"] = _terrain(_gen(seed), [case["points"]], [side], [2], 0.02, 0.06).double() * 0.01
        s["settings"] = engine.CompatSettings(scale=case["scale"], cell_size=2.0, site_radius=5.0, query_radius=4.99,
                                              point_min=0, multiplier=10000, total_ncols=case["ncols"],
                                              total_nrows=case["nrows"])
        s["wp"] = engine.CompatWP(nrows=case["nrows"], ncols=case["ncols"])
        s["h"] = torch.empty(case["nrows"], case["ncols"], dtype=torch.float32, device=DEV)
        s["res"] = torch.empty(case["nrows"], case["ncols"], dtype=torch.int32, device=DEV)
    else:
        raise ValueError(kind)
    return s


def run(s):
    eng, kind = the_engine(), s["kind"]
    st = torch.cuda.current_stream().cuda_stream
    if kind == "call":
        eng.interpolate_device(s["wp"], s["xyz"], s["xyz"].shape[0], s["h"], s["gid"], s["site"], stream=st, stats=False)
        return [s["h"], s["site"]]
    if kind == "batch":
        if s["host"]:
            s["batch"].run(s["xyz"], s["h"], stats=False)
        else:
            s["batch"].run_device(s["xyz"], s["h"], stream=st)
        return [s["h"]]
    if kind == "segment":
        return [eng.segment_run(s["xyz"], *s["args"], out_h=s["h"])[0]]
    if kind == "served":
        srv = s["server"]
        tickets = [srv.submit(x0, y0, k, k, cell, out_h=s["out"][i])
                   for i, (x0, y0, k, cell) in enumerate(s["requests"])]
        return [srv.wait(t)[0] for t in tickets]
    if kind == "spacetime":
        eng.interpolate_spacetime_device(s["wp"], s["xyz"], s["t"], s["xyz"].shape[0], s["h"], 50, s["radius"], 100,
                                         stream=st, stats=False)
        return [s["h"]]
    eng.interpolate_compat_device(s["settings"], s["wp"], s["xyz"], s["xyz"].shape[0], s["h"], s["res"], stream=st)
    return [s["h"], s["res"]]


def work(case):
    """Points read once, outputs written once; a divide and a multiply-add per cell."""
    kind = case["kind"]
    if kind == "batch":
        sp = _specs(case)
        n, cells = sum(s[2] for s in sp), sum(s[0] * s[0] for s in sp)
        return {"bytes": 12 * n + 4 * cells, "flops": 3 * cells}
    if kind == "served":
        rq = _requests(case)
        cells = sum(k * k for _, _, k, _ in rq)
        dens = case["points"] / (case["side_m"] * 100.0) ** 2
        n = sum(dens * (k * c) ** 2 for _, _, k, c in rq)
        return {"bytes": 12 * n + 4 * cells, "flops": 3 * cells}
    n, cells = case["points"], case["ncols"] * case["nrows"]
    b = 12 * n + 4 * cells
    if kind == "call":
        if case["gid"]:
            b += 4 * n
        if case["site"]:
            b += 4 * (case["ncols"] + 2 * case["halo"]) * (case["nrows"] + 2 * case["halo"])
    elif kind == "spacetime":
        b += 4 * n
    elif kind == "compat":
        b = 24 * n + 8 * cells
    return {"bytes": b, "flops": 3 * cells}


# ---------------------------------------------------------------------------
# the same results in 64 bits, without the engine
# ---------------------------------------------------------------------------

_PB = 32           # pixels per side of a block that shares its candidate points


def _isqrt(v):
    r = v.double().sqrt().floor().long()
    r = torch.where(r * r > v, r - 1, r)
    return torch.where((r + 1) * (r + 1) <= v, r + 1, r)


def _nearest(xyz, gid, lift, rx0, ry0, rw, rh, cs):
    """Per raster pixel the least (squared distance + lift, gid) -> (d2, gid),
    int64.  Points near a block of pixels are its candidates: a site known to
    lie near the block bounds how far any pixel's nearest site can be."""
    order = torch.argsort(xyz[:, 1])
    x, y, gid, lift = xyz[order, 0].long(), xyz[order, 1].long(), gid[order], lift[order]
    d_out = torch.empty(rh, rw, dtype=torch.int64, device=DEV)
    g_out = torch.empty(rh, rw, dtype=torch.int64, device=DEV)
    nbx, nby = -(-rw // _PB), -(-rh // _PB)
    cx = (rx0 + torch.arange(nbx, device=DEV) * _PB + (_PB - 1) / 2) * cs
    cy = (ry0 + torch.arange(nby, device=DEV) * _PB + (_PB - 1) / 2) * cs
    # one point of every occupied bucket of 8 x 8 cells
    key = torch.div(y - y.min(), 8 * cs, rounding_mode="floor") * (1 << 20) + torch.div(x - x.min(), 8 * cs,
                                                                                        rounding_mode="floor")
    _, inv = torch.unique(key, return_inverse=True)
    rep = torch.zeros(int(inv.max()) + 1, dtype=torch.int64, device=DEV)
    rep[inv] = torch.arange(x.numel(), device=DEV)
    sx, sy = x[rep].double(), y[rep].double()
    emax = float(lift.max())
    half = _PB / 2 * 1.4143 * cs
    reach = torch.empty(nby, nbx, dtype=torch.float64, device=DEV)
    for b in range(nby):
        best = torch.full((nbx,), math.inf, dtype=torch.float64, device=DEV)
        for k in range(0, sx.numel(), 1 << 17):
            d = (cx[:, None] - sx[None, k:k + (1 << 17)]) ** 2 + (cy[b] - sy[k:k + (1 << 17)]) ** 2
            best = torch.minimum(best, d.min(1).values)
        reach[b] = ((best.sqrt() + half) ** 2 + emax).sqrt() + half + 2
    lo = torch.searchsorted(y, (cy[:, None] - reach).floor().long().reshape(-1)).tolist()
    hi = torch.searchsorted(y, (cy[:, None] + reach).ceil().long().reshape(-1), right=True).tolist()
    reach, cxl = reach.reshape(-1).tolist(), cx.tolist()
    big = torch.tensor(1 << 62, device=DEV)
    for b in range(nbx * nby):
        bx, by = b % nbx, b // nbx
        keep = ((x[lo[b]:hi[b]] - cxl[bx]).abs() <= reach[b]).nonzero()[:, 0] + lo[b]
        qx, qy, qg, ql = x[keep], y[keep], gid[keep], lift[keep]
        i0, i1, j0, j1 = bx * _PB, min(rw, bx * _PB + _PB), by * _PB, min(rh, by * _PB + _PB)
        dx2 = ((rx0 + torch.arange(i0, i1, device=DEV)) * cs)[:, None] - qx[None]
        dx2 = dx2 * dx2 + ql[None]
        rows = max(1, int(3e7 // max(1, dx2.numel())))
        for j in range(j0, j1, rows):
            je = min(j1, j + rows)
            dy = ((ry0 + torch.arange(j, je, device=DEV)) * cs)[:, None] - qy[None]
            d = (dy * dy)[:, None, :] + dx2[None]
            m = d.min(2).values
            d_out[j:je, i0:i1] = m
            g_out[j:je, i0:i1] = torch.where(d == m[:, :, None], qg[None, None], big).min(2).values
    return d_out, g_out


def _spread(Z, C, z, R2, rx0, ry0, ncols, nrows):
    """Adds z and one to every cell within sqrt(R2) of its pixel; Z and C hold
    per-row differences, one column wider than the grid."""
    rw = R2.shape[1]
    r2, order = R2.reshape(-1).sort(descending=True)
    n = int((r2 >= 0).sum())
    r2, order = r2[:n], order[:n]
    px, py, zz = rx0 + order % rw, ry0 + torch.div(order, rw, rounding_mode="floor"), z.reshape(-1)[order]
    asc = -r2
    dy = 0
    while n:
        m = int(torch.searchsorted(asc, torch.tensor(-dy * dy, device=DEV), right=True))
        if m == 0 or dy > 40000:
            break
        w = _isqrt(r2[:m] - dy * dy)
        a, b = (px[:m] - w).clamp(min=0), (px[:m] + w).clamp(max=ncols - 1)
        for sgn in (1, -1) if dy else (1,):
            row = py[:m] + sgn * dy
            ok = ((row >= 0) & (row < nrows) & (a <= b)).nonzero()[:, 0]
            ra, rb, zk = row[ok] * (ncols + 1) + a[ok], row[ok] * (ncols + 1) + b[ok] + 1, zz[ok]
            one = torch.ones_like(zk)
            Z.view(-1).index_add_(0, ra, zk).index_add_(0, rb, -zk)
            C.view(-1).index_add_(0, ra, one).index_add_(0, rb, -one)
        dy += 1


def _heights(Z, C):
    Z, C = Z.cumsum(1)[:, :-1], C.cumsum(1)[:, :-1]
    return torch.where(C > 0, Z.double() / C.clamp(min=1).double() * 0.01, torch.tensor(-9999.0, dtype=torch.float64,
                                                                                        device=DEV))


def _field(ncols, nrows):
    return [torch.zeros(nrows, ncols + 1, dtype=torch.int64, device=DEV) for _ in range(2)]


def _exact_grid(xyz, gid, ncols, nrows, cs, halo=0):
    rx0, rw, rh = -halo, ncols + 2 * halo, nrows + 2 * halo
    d2, g = _nearest(xyz, gid, torch.zeros_like(gid), rx0, rx0, rw, rh, cs)
    zof = torch.empty(int(gid.max()) + 1, dtype=torch.int64, device=DEV)
    zof[gid] = xyz[:, 2].long()
    R2 = torch.div(d2, cs * cs, rounding_mode="floor").clamp(max=rw * rw + rh * rh)
    Z, C = _field(ncols, nrows)
    _spread(Z, C, zof[g], R2, rx0, rx0, ncols, nrows)
    return _heights(Z, C)


def exact(case, seed):
    kind = case["kind"]
    if kind == "call":
        xyz = _call_points(case, seed)
        gid = _call_gid(case, seed).long() if case["gid"] else torch.arange(xyz.shape[0], device=DEV)
        return [_exact_grid(xyz, gid, case["ncols"], case["nrows"], case["cell"], case["halo"]), None]
    if kind == "batch":
        sp = _specs(case)
        if len(sp) > 60 or sum((-(-s[0] // _PB)) ** 2 for s in sp) > 12_000:
            return None                    # too many pixel blocks: far over 20 seconds
        _, xyz, _ = _batch_points(case, seed)
        out, pt = [], 0
        for k, (side, cell, n, _) in enumerate(sp):
            p = xyz[pt:pt + n].clone()
            p[:, :2] -= torch.tensor(synth.tile_origin(k), dtype=torch.int32, device=DEV)
            out.append(_exact_grid(p, torch.arange(n, device=DEV), side, side, cell).reshape(-1))
            pt += n
        return [torch.cat(out)]
    if kind == "segment":
        xyz = _cloud(case, seed, case["ncols"] * case["cell"], case["nrows"] * case["cell"], 0.012, 0.08)
        return [_exact_grid(xyz, torch.arange(xyz.shape[0], device=DEV), case["ncols"], case["nrows"], case["cell"])]
    if kind == "spacetime":
        nc, nr, cs, rt = case["ncols"], case["nrows"], case["cell"], case["radius"]
        xyz = _cloud(case, seed, nc * cs, nr * cs, 0.03, 0.12)
        t = _st_times(case, seed).long()
        Z, C = _field(nc, nr)
        for j in range(-rt, rt + 1):
            at = ((50 + j - t).abs() <= rt).nonzero()[:, 0]
            if at.numel() == 0:
                continue
            lift = ((50 + j - t[at]) * 100) ** 2
            d2, g = _nearest(xyz[at], at, lift, 0, 0, nc, nr, cs)
            e = d2 - (j * 100) ** 2
            R2 = torch.where(e >= 0, torch.div(e.clamp(min=0), cs * cs, rounding_mode="floor"), -1)
            R2 = R2.clamp(max=nc * nc + nr * nr)
            _spread(Z, C, xyz[:, 2].long()[g], R2, 0, 0, nc, nr)
        return [_heights(Z, C)]
    # served: a request's raster is the whole cloud's; compat: float32 plane
    # depths decide each pixel's site, so no 64-bit value exists
    return None
