"""Calls at the edges of the engine's routes, bit for bit against the oracle:
thin tiles without points beside tiles with points, wide cells, scratch limits."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import NATIVE, ROOT

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def eng():
    from terranni_b200 import engine
    e = engine.Engine(device=0)
    yield e
    e.close()


def _same(a, b):
    return np.array_equal(a.view(np.uint32), b.view(np.uint32))


def _points(rng, n, w, h):
    return np.stack([rng.integers(0, w, n), rng.integers(0, h, n), rng.integers(0, 3000, n)], 1).astype(np.int32)


# tiles (ncols, nrows, points): the thin ones have several superblocks of bins
@pytest.mark.parametrize("bin_target", [0, 1])
@pytest.mark.parametrize("shapes", [
    [(170, 1, 0), (64, 48, 3000)],
    [(120, 90, 20000), (1, 300, 0), (512, 1, 0), (300, 2, 500), (2, 300, 0)],
    [(20000, 2, 0), (512, 1, 40), (50, 1, 0), (40, 40, 9000)],
])
def test_batch_with_thin_empty_tiles(eng, oracle, shapes, bin_target):
    from terranni_b200 import engine
    rng = np.random.default_rng(len(shapes) + bin_target)
    rows, tiles, pt, out = [], [], 0, 0
    for nc, nr, n in shapes:
        xyz = _points(rng, n, nc * 100, nr * 100)
        tiles.append(engine.make_tile(engine.make_wp(nc, nr, 100), pt, n, out, out))
        rows.append(xyz)
        pt += n
        out += nc * nr
    xyz = np.concatenate(rows)
    h, site = np.empty(out, np.float32), np.empty(out, np.uint32)
    for order in (False, True):
        with eng.batch(tiles, bin_target=bin_target, order_by_cost=order) as b:
            for _ in range(2):
                h[:], site[:] = 7.0, 7
                b.run(xyz, h, out_site=site)
                o = 0
                for (nc, nr, n), p in zip(shapes, rows):
                    g, s = h[o:o + nc * nr].reshape(nr, nc), site[o:o + nc * nr].reshape(nr, nc)
                    o += nc * nr
                    if n == 0:
                        assert np.all(g == np.float32(-9999.0)) and np.all(s == 0xFFFFFFFF)
                        continue
                    ref = oracle.interpolate(oracle.make_wp(nc, nr, 100), p)
                    assert _same(g, ref["h"]) and np.array_equal(s, ref["site"])


def test_spacetime_transect_with_empty_time_values(eng, oracle):
    from terranni_b200 import engine
    rng = np.random.default_rng(4)
    for nc, nr in ((512, 1), (1, 400)):
        xyz = _points(rng, 9000, nc * 100, nr * 100)
        t = rng.choice(np.array([-2, 0, 1]), 9000).astype(np.int32)      # of the values -2 .. 2, two have no point
        ref = oracle.interpolate_spacetime(oracle.make_wp(nc, nr, 100), xyz, t, 0, 1, 120)
        h, _ = eng.interpolate_spacetime(engine.make_wp(nc, nr, 100), xyz, t, 0, 1, 120)
        assert _same(h, ref["h"])


def test_segment_row_with_empty_tiles(eng, oracle):
    rng = np.random.default_rng(6)
    xyz = _points(rng, 12000, 100_000, 100)
    xyz[6000:, 0] += 200_000                            # cells 1000 to 2000 hold no point
    ref = oracle.interpolate(oracle.make_wp(3000, 1, 100), xyz)
    for halo in (2, 0):
        h, site, st = eng.segment_run(xyz, 3000, 1, 100, tile=250, halo=halo, tiles_per_batch=6, site=True)
        assert _same(h, ref["h"]) and np.array_equal(site, ref["site"])


# rings of points around pixels that lie more than 2^24 units apart: nearest and
# next differ by a unit or less, and the far pass's float filter works on offsets
# that round by several.  The pixels between hold a point each and are settled
# before, so that a ring's pixel is alone in its eighth of the group.
@pytest.mark.parametrize("cell,count", [(3_000_000, 32), (10_000_000, 8), (15_000_000, 8), (10_000_000, 32)])
def test_far_pass_on_wide_cells(oracle, cell, count):
    from terranni_b200 import engine
    rng = np.random.default_rng(cell + count)
    n = 320_000 // count
    rows = []
    for k in range(0, count, 4):
        a, rad = rng.uniform(0, 2 * np.pi, n), rng.uniform(40_000, 40_004, n)
        rows.append(np.stack([k * cell + rad * np.cos(a), rad * np.sin(a), rng.integers(0, 3000, n)], 1))
        rows.append(np.stack([(k + np.arange(1, 4)) * cell, np.zeros(3), rng.integers(0, 3000, 3)], 1))
    xyz = np.rint(np.concatenate(rows)).astype(np.int32)
    ref = oracle.interpolate(oracle.make_wp(count, 1, cell), xyz)
    with engine.Engine(device=0, bin_target=1) as e:
        h, site, st = e.interpolate(engine.make_wp(count, 1, cell), xyz, site=True)
        assert st.evals_far > 0
    assert np.array_equal(site, ref["site"]) and _same(h, ref["h"])
    tile = engine.make_tile(engine.make_wp(count, 1, cell), 0, xyz.shape[0], 0, 0,
                            extent=(*xyz[:, :2].min(0).tolist(), *xyz[:, :2].max(0).tolist()))
    with engine.Engine(device=0) as e, e.batch([tile], bin_target=1, far_group=1) as b:     # groups in pixel rows
        h, site = np.empty((1, count), np.float32), np.empty((1, count), np.uint32)
        b.run(xyz, h.reshape(-1), out_site=site.reshape(-1))
    assert np.array_equal(site, ref["site"]) and _same(h, ref["h"])


def _budget_calls():
    """Calls whose grouped points (or gathered records) need more room than the
    rest of their scratch: name -> (call on an engine -> heights)."""
    from terranni_b200 import engine
    rng = np.random.default_rng(12)
    xyz = _points(rng, 60000, 6400, 6400)
    wp = engine.make_wp(64, 64, 100)
    times = rng.integers(-3, 4, 60000).astype(np.int32)
    big = np.concatenate([_points(rng, 300_000, 9600, 9600) + np.array([k * 20000, 0, 0], np.int32) for k in range(15)])
    world = np.stack([rng.uniform(0, 80, 30000), rng.uniform(0, 60, 30000), rng.uniform(0, 30, 30000)], 1)
    cset = engine.CompatSettings(scale=2, cell_size=2.0, site_radius=5.0, query_radius=4.99, point_min=0, multiplier=10000,
                                 total_ncols=40, total_nrows=30)

    def batch(e, tiles, rows, cells, graph):
        out = np.empty(cells, np.float32)
        with e.batch(tiles, use_graph=graph) as b:
            for _ in range(2):
                out[:] = 5.0
                b.run(rows, out)
        return out

    def two_kinds(e):
        # a batch keeps its scratch while other calls come and go beside it
        out = np.empty(64 * 64, np.float32)
        with e.batch([engine.make_tile(wp, 0, 60000, 0)], use_graph=True) as b:
            b.run(xyz, out)
            h = e.interpolate(wp, xyz, site=True)[0]
            assert _same(h.reshape(-1), out)
            out[:] = 5.0
            b.run(xyz, out)
        return out

    return {
        "single": lambda e: e.interpolate(wp, xyz, site=True)[0],
        "batch": lambda e: batch(e, [engine.make_tile(wp, 0, 60000, 0)], xyz, 64 * 64, False),
        "batch_graph": lambda e: batch(e, [engine.make_tile(wp, 0, 60000, 0)], xyz, 64 * 64, True),
        "batch_slices": lambda e: batch(e, [engine.make_tile(engine.make_wp(96, 96, 100, k * 20000, 0), k * 300_000, 300_000,
                                                             k * 9216) for k in range(15)], big, 15 * 9216, False),
        "two_kinds": two_kinds,
        "segment": lambda e: e.segment_run(xyz, 64, 64, 100, tile=32, halo=6, tiles_per_batch=1)[0],
        "spacetime": lambda e: e.interpolate_spacetime(wp, xyz, times, 0, 1, 100)[0],
        "compat": lambda e: e.interpolate_compat(cset, engine.CompatWP(nrows=30, ncols=40), world)[0],
    }


# the room that only speeds a call up never costs another allocation its place:
# every budget above the smallest accepted one is accepted, with the same bits
@pytest.mark.parametrize("kind", ["single", "batch", "batch_graph", "batch_slices", "two_kinds", "segment", "spacetime",
                                  "compat"])
def test_no_budget_is_refused_above_an_accepted_one(eng, kind):
    from terranni_b200 import engine
    call = _budget_calls()[kind]
    want = call(eng).copy()

    def accepted(budget):
        with engine.Engine(device=0, mem_budget=budget) as e:
            try:
                got = call(e)
            except engine.DnniError as err:
                assert err.status == 2
                return False
        assert _same(got, want)
        return True

    lo, hi = 1, 1 << 30
    assert accepted(hi) and not accepted(lo)
    while hi - lo > 256:
        mid = (lo + hi) // 2
        if accepted(mid):
            hi = mid
        else:
            lo = mid
    for k in range(1, 49):
        assert accepted(int(hi * 1.025 ** k))


# groups beyond 32-bit distances against the same geometry in smaller units: few
# groups, groups that leave their warp, and a list long enough that they stay
@pytest.mark.parametrize("side,n,scale", [(60, 900, 500), (300, 90_000, 50), (300, 9000, 50_000), (800, 120_000, 50),
                                          (800, 30_000, 50_000)])
@pytest.mark.parametrize("groups", [1, 2])
def test_far_pass_beyond_32_bits(eng, side, n, scale, groups):
    from terranni_b200 import engine
    rng = np.random.default_rng(side + n)
    w = 20 * side
    xyz = _points(rng, n, w, w)
    d = (xyz[:, :2] - w // 2).astype(np.int64)
    xyz = xyz[(d * d).sum(1) > (0.46 * w) ** 2]
    out = []
    for k in (1, scale):
        p = xyz * np.array([k, k, 1], np.int32)
        tile = engine.make_tile(engine.make_wp(side, side, 20 * k), 0, p.shape[0], 0, 0, extent=(0, 0, w * k - 1, w * k - 1))
        h, site = np.empty(side * side, np.float32), np.empty(side * side, np.uint32)
        with eng.batch([tile], far_group=groups) as b:
            b.run(p, h, out_site=site)
        out.append((h, site))
    assert np.array_equal(out[0][1], out[1][1]) and _same(out[0][0], out[1][0])


def test_a_request_by_itself_does_not_wait_for_company():
    """While a long batch runs and a slot is free, a request that comes alone is
    launched at once."""
    import time
    from terranni_b200 import engine
    rng = np.random.default_rng(3)
    xyz = _points(rng, 400_000, 120_000, 120_000)
    idle, queued = [], []
    with engine.Engine(device=0) as e, e.server(xyz, slots=2, slot_bytes=4 << 30) as srv:
        for _ in range(16):
            idle.append(srv.wait(srv.submit(0, 0, 64, 64, 100))[2]["ms_queue"])
            time.sleep(0.002)
            long = srv.submit(0, 0, 6000, 6000, 20)
            time.sleep(0.002)
            h, _, r = srv.wait(srv.submit(10_000, 20_000, 64, 64, 100))
            queued.append(r["ms_queue"])
            srv.wait(long)
            time.sleep(0.002)
    assert min(queued) < min(idle) + 0.05


def test_a_slot_has_no_room_to_spare_for_the_gather_list():
    """The smallest slot that takes a request over the whole cloud does not depend
    on how many buckets, and so gather chunks, the cloud has."""
    from terranni_b200 import engine
    rng = np.random.default_rng(5)
    xyz = _points(rng, 60_000, 40_000, 40_000)

    def fits(bucket, bytes_):
        with engine.Engine(device=0) as e, e.server(xyz, bucket=bucket, slots=1, slot_bytes=bytes_) as srv:
            try:
                srv.wait(srv.submit(0, 0, 100, 100, 400))
            except engine.DnniError as err:
                assert err.status == 2
                return False
            return True

    least = []
    for bucket in (40_000, 100):
        lo, hi = 1 << 12, 1 << 26
        while hi - lo > 256:                # a slot takes a quarter more than it is asked for
            mid = (lo + hi) // 2
            lo, hi = (lo, mid) if fits(bucket, mid) else (mid, hi)
        least.append(hi)
    assert least[1] <= least[0] + 256


# site squares over the whole raster and far beyond it: the count of tiles that one
# reaches has to stay within what the raster has
@pytest.mark.parametrize("site_radius", [1e4, 2.5e10, 1e11, 1e12, 1e14])
def test_compat_squares_beyond_the_raster(eng, oracle, site_radius):
    from terranni_b200 import engine
    rng = np.random.default_rng(2)
    nc, nr, n = 40, 30, 60
    pts = np.stack([rng.uniform(0, 2 * nc, n), rng.uniform(0, 2 * nr, n), rng.uniform(0, 30, n)], 1)
    arg = dict(scale=5, cell_size=2.0, site_radius=site_radius, query_radius=4.99, point_min=0, multiplier=10000,
               total_ncols=nc, total_nrows=nr)
    ref_h, ref_res = oracle.compat(oracle.CompatSettings(**arg), oracle.CompatWP(nrows=nr, ncols=nc), pts)
    h, res = eng.interpolate_compat(engine.CompatSettings(**arg), engine.CompatWP(nrows=nr, ncols=nc), pts)
    assert np.array_equal(res, ref_res) and _same(h, ref_h)


@pytest.fixture(scope="module")
def span():
    src, so = os.path.join(NATIVE, "dnni_span.cu"), os.path.join(NATIVE, "libdnni_span.so")
    csrc = os.path.join(ROOT, "terranni_b200", "csrc")
    deps = [src] + [os.path.join(csrc, f) for f in ("dnni_search.cuh", "dnni_kernels.cuh", "dnni_plan.h")]
    if not os.path.exists(so) or any(os.path.getmtime(d) > os.path.getmtime(so) for d in deps):
        subprocess.run(["/usr/local/cuda/bin/nvcc", "-O3", "-std=c++17", "-Xcompiler", "-fPIC", "-shared", "-gencode",
                        "arch=compute_100a,code=sm_100a", "-o", so, src], check=True, capture_output=True)
    return ctypes.CDLL(so)


# the estimate's exact range, R2 - dy^2 of every value below 2^20, and samples of
# the corrected estimate beyond it up to the largest R2
@pytest.mark.parametrize("n0,step,dy,n", [(0, 1, 0, 1 << 20), (0, 1, 1, (1 << 20) - 1), (0, 1, 511, (1 << 20) - 511 ** 2),
                                          (0, 1, 1023, (1 << 20) - 1023 ** 2), (1 << 20, 1, 0, 1 << 22),
                                          (0, 4093, 30000, 300_000), (1 << 20, 2039, 0, 1_050_000)])
def test_half_widths_are_exact(span, n0, step, dy, n):
    out = np.empty(n, np.int32)
    assert span.span_half_widths(ctypes.c_int64(n0), ctypes.c_int64(step), dy, n, out.ctypes.data_as(ctypes.c_void_p)) == 0
    v = n0 + np.arange(n, dtype=np.int64) * step
    assert int(v[-1]) + dy * dy < 1 << 31
    w = np.floor(np.sqrt(v.astype(np.float64))).astype(np.int64)
    assert np.all(w * w <= v) and np.all((w + 1) ** 2 > v) and np.array_equal(out, w)
