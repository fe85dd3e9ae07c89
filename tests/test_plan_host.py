"""The batch plan (host build of the engine's planning code; no GPU)."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import NATIVE, ROOT

SO = os.path.join(NATIVE, "libdnni_edge.so")


@pytest.fixture(scope="module")
def edge():
    src = os.path.join(NATIVE, "dnni_edge.cu")
    csrc = os.path.join(ROOT, "terranni_b200", "csrc")
    deps = [src] + [os.path.join(csrc, f) for f in ("dnni_search.cuh", "dnni_kernels.cuh", "dnni_plan.h")]
    if not os.path.exists(SO) or any(os.path.getmtime(d) > os.path.getmtime(SO) for d in deps):
        subprocess.run(["/usr/local/cuda/bin/nvcc", "-O2", "-std=c++17", "-Xcompiler", "-fPIC", "-shared", "-gencode",
                        "arch=compute_100a,code=sm_100a", "-o", SO, src], check=True, capture_output=True)
    return ctypes.CDLL(SO)


def _regions(edge, shapes, points, target):
    n = len(shapes)
    nc, nr = (np.array([s[k] for s in shapes], np.int32) for k in (0, 1))
    pts = np.array(points, np.int64)
    strips, whole, bins = (np.zeros(n, np.int64) for _ in range(3))
    most = ctypes.c_int32(0)
    p = lambda a: a.ctypes.data_as(ctypes.c_void_p)
    assert edge.edge_batch_regions(n, p(nc), p(nr), 100, p(pts), ctypes.c_double(target), p(strips), p(whole), p(bins),
                                   ctypes.byref(most)) == 0
    return strips, whole, bins, most.value


# thin tiles, whose bin grid has several superblocks even without points
@pytest.mark.parametrize("target", [1.0, 4.0])
@pytest.mark.parametrize("shape", [(170, 1), (512, 1), (1, 300), (20000, 2), (50, 1), (64, 64), (32767, 1)])
def test_tiles_without_points_list_no_region(edge, shape, target):
    strips, whole, bins, most = _regions(edge, [shape, (40, 40), shape], [0, 900, 20000], target)
    assert strips[0] == 0 and whole[0] == 0
    assert (strips[1], whole[1]) == (0, 1)           # few points on one superblock: one region
    assert strips[2] * 512 + whole[2] * 4096 == bins[2]
    assert most == max(1, strips[2], whole[2])
    assert _regions(edge, [shape], [0], target)[3] == 1
