"""The search's float quotient estimates against integer division, over their
stated ranges and at their edges, and the binning plan's region limits (host
build of the same code; no GPU)."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import NATIVE, ROOT

SO = os.path.join(NATIVE, "libdnni_est.so")


@pytest.fixture(scope="module")
def est():
    src = os.path.join(NATIVE, "dnni_est.cu")
    deps = [src] + [os.path.join(ROOT, "terranni_b200", "csrc", f) for f in ("dnni_search.cuh", "dnni_kernels.cuh",
                                                                            "dnni_plan.h")]
    if not os.path.exists(SO) or any(os.path.getmtime(d) > os.path.getmtime(SO) for d in deps):
        subprocess.run(["/usr/local/cuda/bin/nvcc", "-O2", "-std=c++17", "-Xcompiler", "-fPIC", "-shared", "-gencode",
                        "arch=compute_100a,code=sm_100a", "-o", SO, src], check=True, capture_output=True)
    L = ctypes.CDLL(SO)
    L.est_eval.argtypes = [ctypes.c_int] + [ctypes.c_void_p] * 3 + [ctypes.c_int64, ctypes.c_void_p]
    L.est_regions.argtypes = [ctypes.c_int64, ctypes.c_int32, ctypes.c_int32, ctypes.c_double, ctypes.c_void_p]

    def run(kind, x, u, v=None):
        x, u = np.ascontiguousarray(x, np.uint32), np.ascontiguousarray(u, np.uint32)
        v = np.zeros_like(x) if v is None else np.ascontiguousarray(v, np.uint32)
        out = np.empty(x.size, np.int64)
        L.est_eval(kind, x.ctypes.data, u.ctypes.data, v.ctypes.data, x.size, out.ctypes.data)
        return out
    run.lib = L
    return run


def _around(q, u, most):
    """x = q u + {-1, 0, 1, u - 1}, inside [0, most)."""
    q, u = q.astype(np.int64), u.astype(np.int64)
    x = np.concatenate([q * u + d for d in (-1, 0, 1)] + [q * u + u - 1])
    u = np.concatenate([u] * 4)
    ok = (x >= 0) & (x < most)
    return x[ok], u[ok]


@pytest.mark.parametrize("kind,most,qmost", [(0, 1 << 22, 1 << 22), (1, 3 << 30, 1 << 20)])
def test_floor_quotients(est, kind, most, qmost):
    r = np.random.default_rng(kind)
    u = np.exp(r.uniform(0, np.log(1 << 24), 200_000)).astype(np.int64) + 1
    q = (r.random(u.size) * np.minimum(most // u + 1, qmost - 1)).astype(np.int64)
    x, u = _around(q, u, most)
    ok = x // u < qmost
    x, u = x[ok], u[ok]
    assert np.array_equal(est(kind, x, u), x // u)


def test_r2_quotient_and_cap(est):
    r = np.random.default_rng(3)
    cs = np.concatenate([np.exp(r.uniform(0, np.log(32767), 200_000)).astype(np.int64) + 0, [1, 2, 100, 32767]])
    q = np.exp(r.uniform(0, np.log(1 << 31), cs.size)).astype(np.int64)
    x, cs2 = _around(np.minimum(q, (1 << 31) // (cs * cs)), cs * cs, 1 << 31)
    cs = np.sqrt(cs2.astype(np.float64)).round().astype(np.int64)
    cap = r.integers(0, 1 << 31, x.size)
    assert np.array_equal(est(2, x, cs, cap), np.minimum(x // cs2, cap))


@pytest.mark.parametrize("n,w,h,target", [
    (1, 100, 100, 4), (8192, 5000, 5000, 4), (8193, 5000, 5000, 4), (8192, 1 << 29, 3, 4), (200_000, 51200, 51200, 4),
    (20_000_000, 409600, 409600, 4), (40_000_000, 409600, 409600, 4), (300_000_000, 1 << 20, 1 << 20, 1),
    (1 << 30, 1 << 29, 1 << 10, 1), (50_000_000, 1 << 29, 64, 1),
])
def test_regions_stay_within_a_chunks_histogram(est, n, w, h, target):
    out = np.zeros(5, np.int64)
    assert est.lib.est_regions(n, w, h, float(target), out.ctypes.data) == 0
    rsh, regions, bins, most, band = out.tolist()
    assert rsh in (9, 12) and regions << rsh == bins
    assert regions <= most                    # one shared-memory counter each
    assert 3 * regions + 1 <= bins            # the region arrays fit the bin counts
    assert band in (8, 16, 32, 64)
    if regions == 1:
        assert n <= 8192
