"""The far pass's filter of candidate points (host build of the engine's code;
no GPU): a point that lies on a pixel's bound is never left out, however large
the group and the circle."""
import ctypes

import numpy as np
import pytest

from test_plan_host import edge  # noqa: F401  (fixture)


# largest offset of a group's pixels from its corner: 8 or 32 cells of up to 2^30 units together
@pytest.mark.parametrize("most", [1 << 10, 1 << 16, 1 << 22, 1 << 24, 1 << 25, 1 << 27, 1 << 30])
@pytest.mark.parametrize("layout", ["square", "row"])
def test_a_point_on_the_bound_is_kept(edge, most, layout):  # noqa: F811
    r = np.random.default_rng(most + len(layout))
    n = 300_000
    cells = 8 if layout == "square" else 32
    cs = np.maximum(1, np.exp(r.uniform(np.log(most / 16), np.log(most), n)).astype(np.int64) // cells)
    base = r.integers(0, cells // (2 if layout == "square" else 4), n)
    dx = np.array([0, 1, 0, 1] if layout == "square" else [0, 1, 2, 3])
    dy = np.array([0, 0, 1, 1] if layout == "square" else [0, 0, 0, 0])
    px = ((2 if layout == "square" else 4) * base[:, None] + dx) * cs[:, None]
    py = ((2 * r.integers(0, 2, n))[:, None] + dy) * cs[:, None] if layout == "square" else np.zeros_like(px)
    act = r.random((n, 4)) < 0.5
    own = r.integers(0, 4, n)
    act[np.arange(n), own] = True
    rad = np.exp(r.uniform(np.log(1), np.log(1 << 26), n))
    a = r.uniform(0, 2 * np.pi, n)
    a[::7] = np.round(a[::7] / (np.pi / 2)) * (np.pi / 2)
    ox, oy = px[np.arange(n), own], py[np.arange(n), own]
    qx, qy = ox + np.rint(rad * np.cos(a)).astype(np.int64), oy + np.rint(rad * np.sin(a)).astype(np.int64)
    d2 = np.zeros((n, 4), np.int64)
    d2[np.arange(n), own] = (qx - ox) ** 2 + (qy - oy) ** 2
    hit = np.zeros(n, np.uint8)
    act8 = np.ascontiguousarray(act, np.uint8)
    ext = (cells - 1) * cs
    edge.edge_circle(ctypes.c_int64(n), *(np.ascontiguousarray(v).ctypes.data_as(ctypes.c_void_p)
                                         for v in (px, py, act8, d2, ext, qx, qy)), hit.ctypes.data_as(ctypes.c_void_p))
    assert hit.all()
