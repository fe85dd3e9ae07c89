"""The engine's size-dependent routes at their edges: binning from one block,
by strips, by superblocks and without room for the grouped points; the far
pass by warps and by whole CTAs, in 32 and 64 bits; span rows beyond 1024 cells;
finalize segments with packed, unpacked and wide values; the reference-default
site pass with and without room for its records.  All results are exact, so
every comparison is bit for bit: against the oracle where it is quick, else
against the same work through another route."""
import numpy as np
import pytest

from conftest import terrain_case

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def eng():
    from terranni_b200 import engine
    e = engine.Engine(device=0)
    yield e
    e.close()


def _same(a, b):
    return np.array_equal(a.view(np.uint32), b.view(np.uint32))


def _check(eng, oracle, wp_args, xyz, gid=None, **kw):
    from terranni_b200 import engine
    ref = oracle.interpolate(oracle.make_wp(*wp_args, **kw), xyz, gid)
    h, site, st = eng.interpolate(engine.make_wp(*wp_args, **kw), xyz, gid, site=True)
    assert np.array_equal(site, ref["site"])
    assert _same(h, ref["h"])
    return st


# one region up to 8192 points on one superblock; chunks of 2048 points (4096 from 2 Mi on); strips
@pytest.mark.parametrize("n", [1, 31, 2047, 2049, 4097, 8191, 8192, 8193, 20481, 70001])
def test_binning_by_point_count(eng, oracle, n):
    rng = np.random.default_rng(n)
    xyz = np.stack([rng.integers(-300, 10300, n), rng.integers(-200, 7000, n), rng.integers(0, 3000, n)], 1).astype(np.int32)
    _check(eng, oracle, (97, 66, 100), xyz)


# all points in one bin, in one row of bins, and evenly spread: regions of very uneven size
@pytest.mark.parametrize("kind", ["bin", "row", "even"])
def test_uneven_regions(eng, oracle, kind):
    rng = np.random.default_rng(5)
    n = 30000
    xyz = np.stack([rng.integers(0, 12800, n), rng.integers(0, 12800, n), rng.integers(0, 3000, n)], 1).astype(np.int32)
    if kind != "even":
        xyz[100:, 1] = 6400
    if kind == "bin":
        xyz[100:, 0] = 6400 + rng.integers(0, 3, n - 100)
    _check(eng, oracle, (128, 128, 100), xyz)


@pytest.mark.parametrize("n,bin_target", [(2_200_000, 1), (2_200_000, 12)])
def test_many_regions_equal_few(eng, n, bin_target):
    """Superblocks against strips, large chunks: the bin size changes the
    route, never the result."""
    from terranni_b200 import engine
    rng = np.random.default_rng(n)
    xyz = np.stack([rng.integers(0, 60000, n), rng.integers(0, 60000, n), rng.integers(0, 3000, n)], 1).astype(np.int32)
    wp = engine.make_wp(600, 600, 100)
    h, site, _ = eng.interpolate(wp, xyz, site=True)
    with engine.Engine(device=0, bin_target=bin_target) as e:
        h2, site2, _ = e.interpolate(wp, xyz, site=True)
    assert np.array_equal(site, site2) and _same(h, h2)


def test_scratch_limit_takes_the_direct_binning(eng, oracle):
    """Dense points on a small grid: the grouped points need more room than
    the late arrays.  Shrinking budgets cross from one binning to the other and
    then refuse; every accepted call gives the same bits."""
    from terranni_b200 import engine
    rng = np.random.default_rng(8)
    n = 60000
    xyz = np.stack([rng.integers(0, 6400, n), rng.integers(0, 6400, n), rng.integers(0, 3000, n)], 1).astype(np.int32)
    wp = engine.make_wp(64, 64, 100)
    want, site, _ = eng.interpolate(wp, xyz, site=True)
    ok = refused = 0
    for budget in range(6_000_000, 1_000_000, -100_000):
        with engine.Engine(device=0, mem_budget=budget) as e:
            try:
                h, s, _ = e.interpolate(wp, xyz, site=True)
            except engine.DnniError as err:
                assert err.status == 2
                refused += 1
                continue
        ok += 1
        assert _same(h, want) and np.array_equal(s, site)
    assert ok and refused


# an empty disc in the middle of a ring of points: few groups (whole CTAs take
# all), more than 592 of them, row groups; cells large enough for 64-bit bounds
@pytest.mark.parametrize("side,cell,n,groups", [(100, 100, 9000, 0), (128, 50, 4000, 0), (161, 100, 30000, 0),
                                                (300, 100, 90000, 0), (161, 100, 30000, 1), (140, 2000, 9000, 0),
                                                (120, 100000, 900, 0)])
def test_far_pass_over_an_empty_disc(eng, oracle, side, cell, n, groups):
    from terranni_b200 import engine
    rng = np.random.default_rng(side + n)
    w = side * cell
    xyz = np.stack([rng.integers(0, w, n), rng.integers(0, w, n), rng.integers(0, 3000, n)], 1).astype(np.int64)
    d = xyz[:, :2] - w // 2
    xyz = xyz[(d * d).sum(1) > (0.42 * w) ** 2].astype(np.int32)
    if not groups:
        _check(eng, oracle, (side, side, cell), xyz)
        return
    ref = oracle.interpolate(oracle.make_wp(side, side, cell), xyz)
    out = np.empty(side * side, np.float32)
    tile = engine.make_tile(engine.make_wp(side, side, cell), 0, xyz.shape[0], 0, extent=(0, 0, w, w))
    with eng.batch([tile], far_group=groups) as b:
        b.run(xyz, out)
    assert _same(out.reshape(side, side), ref["h"])


# half-widths past the estimate's exact range (R2 >= 2^20) and up to its edge
@pytest.mark.parametrize("ncols,nrows", [(1030, 5), (1500, 3), (1023, 40)])
def test_span_rows_of_large_discs(eng, oracle, ncols, nrows):
    _check(eng, oracle, (ncols, nrows, 100), np.array([[3, 2, 500], [ncols * 100 - 7, 90, 900]], np.int32))


# column segments (few bands) with ragged ends, a raster halo, and the three
# forms of a cell's sums: one word, wide values, separate counts
@pytest.mark.parametrize("ncols,nrows,zmax", [(31, 1, 3000), (33, 17, 3000), (65, 16, 3000), (700, 20, 3000),
                                              (700, 20, 40_000_000), (500, 33, 900_000_000)])
def test_finalize_segments(oracle, ncols, nrows, zmax):
    from terranni_b200 import engine
    rng = np.random.default_rng(ncols + nrows)
    n = max(40, ncols * nrows // 3)
    xyz = np.stack([rng.integers(-500, ncols * 100 + 500, n), rng.integers(-500, nrows * 100 + 500, n),
                    rng.integers(-zmax, zmax, n)], 1).astype(np.int32)
    xyz = xyz[(np.abs(xyz[:, 0] - ncols * 50) > ncols * 8)]
    for rs in (1, 3, 6):
        with engine.Engine(device=0, small_radius=rs) as e:
            _check(e, oracle, (ncols, nrows, 100), xyz, raster=(-4, -3, ncols + 5, nrows + 2))


# duplicate ids: the smallest z of equal (distance, id) wins on every route
@pytest.mark.parametrize("n", [500, 9000])
def test_duplicate_ids(eng, oracle, n):
    rng = np.random.default_rng(n)
    xyz = np.stack([rng.integers(0, 64, n) * 100, rng.integers(0, 64, n) * 100, rng.integers(0, 3000, n)], 1).astype(np.int32)
    _check(eng, oracle, (64, 64, 100), xyz, np.full(n, 7, np.uint32))


# time radii held in registers (up to 3) and not; wide values in the stencil
@pytest.mark.parametrize("rt,zmax", [(0, 3000), (3, 3000), (4, 3000), (1, 60_000_000)])
def test_spacetime_routes(eng, oracle, rt, zmax):
    from terranni_b200 import engine
    rng = np.random.default_rng(rt + zmax)
    n, nc, nr = 3000, 71, 40
    xyz = np.stack([rng.integers(0, nc * 100, n), rng.integers(0, nr * 100, n), rng.integers(-zmax, zmax, n)], 1).astype(np.int32)
    t = rng.integers(-2 * rt - 1, 2 * rt + 2, n).astype(np.int32)
    ref = oracle.interpolate_spacetime(oracle.make_wp(nc, nr, 100), xyz, t, 0, rt, 120)
    h, _ = eng.interpolate_spacetime(engine.make_wp(nc, nr, 100), xyz, t, 0, rt, 120)
    assert _same(h, ref["h"])


# squares within one tile of pixels and over several, ragged rasters; then
# budgets that leave no room for the records
@pytest.mark.parametrize("scale,sr,ncols,nrows,n", [(1, 3.0, 31, 33, 900), (5, 5.0, 13, 14, 700), (5, 30.0, 9, 20, 150),
                                                    (2, 60.0, 40, 17, 60), (1, 2.0, 5, 5, 0)])
def test_compat_routes(eng, oracle, scale, sr, ncols, nrows, n):
    from terranni_b200 import engine
    rng = np.random.default_rng(ncols * nrows)
    pts = np.stack([rng.uniform(-5, ncols * 2 + 5, n), rng.uniform(-5, nrows * 2 + 5, n), rng.uniform(0, 30, n)], 1)
    if n:
        pts[n // 2:n // 2 + 20, :2] = pts[:20, :2]           # equal depths: the later draw wins
    arg = dict(scale=scale, cell_size=2.0, site_radius=sr, query_radius=4.99, point_min=0, multiplier=10000,
               total_ncols=ncols, total_nrows=nrows)
    ref_h, ref_res = oracle.compat(oracle.CompatSettings(**arg), oracle.CompatWP(nrows=nrows, ncols=ncols), pts)
    se, we = engine.CompatSettings(**arg), engine.CompatWP(nrows=nrows, ncols=ncols)
    h, res = eng.interpolate_compat(se, we, pts)
    assert np.array_equal(res, ref_res) and _same(h, ref_h)
    ok = refused = 0
    top = 24 * n + 16 * (ncols * scale + 40) * (nrows * scale + 40) + 40 * n + 65536
    for k in range(40, 0, -1):
        with engine.Engine(device=0, mem_budget=max(1, top * k // 40)) as e:
            try:
                h, res = e.interpolate_compat(se, we, pts)
            except engine.DnniError as err:
                assert err.status == 2
                refused += 1
                continue
        ok += 1
        assert np.array_equal(res, ref_res) and _same(h, ref_h)
    assert ok and refused
