"""The mesh build's overlap filter (csrc/tri_box.cuh), compiled for the host
by tests/host_tri_box.cpp, against the exact triangle/box test it stands in
front of: wherever the filter decides, it has to decide as the exact test
does; elsewhere the build runs the exact test."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


@pytest.fixture(scope="module")
def host_filter(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("host_tri_box") / "libhost_tri_box.so")
    subprocess.run(["g++", "-O2", "-ffp-contract=off", "-std=c++17", "-shared", "-fPIC",
                    "-I", os.path.join(ROOT, "sparse-voxel-octrees_gb300", "csrc"),
                    os.path.join(HERE, "host_tri_box.cpp"), "-o", so], check=True)
    L = ctypes.CDLL(so)
    vp = ctypes.c_void_p
    L.host_filter.restype = None
    L.host_filter.argtypes = [vp, ctypes.c_int64, vp, vp, vp, ctypes.c_float, vp]

    def run(tris, centres, half):
        tris = np.ascontiguousarray(tris, np.float32).reshape(-1, 9)
        c = [np.ascontiguousarray(x, np.float32) for x in centres]
        n = np.zeros(4, np.int64)
        L.host_filter(tris.ctypes.data, tris.shape[0], c[0].ctypes.data, c[1].ctypes.data, c[2].ctypes.data,
                      float(half), n.ctypes.data)
        return n

    return run


def triangles(kind, n, side, origin, rng):
    """n triangles around the brick at voxel `origin`, coordinates in voxels
    turned into the unit cube's by 1 / side."""
    c = origin + rng.uniform(0, 8, (n, 1, 3))
    if kind == "small":
        v = c + rng.normal(0, 1.5, (n, 3, 3))
    elif kind == "medium":
        v = c + rng.normal(0, 8, (n, 3, 3))
    elif kind == "large":
        v = c + rng.normal(0, side / 4, (n, 3, 3))
    elif kind == "sliver":
        a = rng.normal(0, 4, (n, 1, 3))
        v = c + a * np.array([0, 1, 0.5])[None, :, None] + rng.normal(0, 1e-4, (n, 3, 3))
    elif kind == "on_planes":  # vertices on voxel faces, edges and corners
        v = np.round(c + rng.normal(0, 3, (n, 3, 3)))
    elif kind == "axis_aligned":  # in a plane of the grid
        v = np.round(c + rng.normal(0, 3, (n, 3, 3)))
        k = rng.integers(0, 3, n)
        v[np.arange(n), :, k] = v[np.arange(n), :1, k]
    elif kind == "half_voxels":
        v = np.round(2 * (c + rng.normal(0, 3, (n, 3, 3)))) / 2
    elif kind == "collinear":
        a = np.round(rng.normal(0, 3, (n, 1, 3)))
        v = np.round(c) + a * np.array([0, 1, 2])[None, :, None]
    else:  # points, and vertices that are not finite
        v = np.repeat(c, 3, 1)
        v[::3, 1] = np.inf
        v[1::3, 2, 0] = np.nan
    return (v / side).astype(np.float32)


@pytest.mark.parametrize("side", [5, 60, 1020, 8188])
@pytest.mark.parametrize("kind", ["small", "medium", "large", "sliver", "on_planes", "axis_aligned", "half_voxels",
                                  "collinear", "degenerate"])
def test_filter_agrees_with_exact_test(host_filter, kind, side):
    rng = np.random.default_rng([side, len(kind)])
    h = np.float32(1) / np.float32(side)
    half = np.float32(0.5) * h
    total = np.zeros(4, np.int64)
    for origin in (np.zeros(3), rng.integers(0, max(1, side - 8), 3), np.full(3, max(0, side - 8))):
        centres = []
        for k in range(3):  # running sums from a start up to a sub-block away
            lo = max(0, int(origin[k]) - int(rng.integers(0, 256)))
            c, row = (np.float32(lo) - np.float32(0.5)) * h, []
            for i in range(lo, int(origin[k]) + 8):
                row.append(c)
                c = np.float32(c + h)
            centres.append(np.array(row[-8:], np.float32))
        total += host_filter(triangles(kind, 1500, side, origin, rng), centres, half)
    seen, decided, wrong, hits = total
    assert wrong == 0
    if kind in ("small", "medium"):  # the build's own triangles: the exact test stays rare
        assert hits > 0 and decided > 0.99 * seen
