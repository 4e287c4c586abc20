"""The one-launch bisection called directly, against the host's decisions made cluster by
cluster: which levels it takes, trees past 46341 points a line and of a box of 2^32 cells,
one block and several, and its three ways out (the limits of a level, too few nodes, a wait
that runs out), after which the host bisects by waves."""
import ctypes
import subprocess
import tempfile

import numpy as np
import pytest

import configs  # noqa: F401  (puts the repository on the path)
from amrclaw_b200.build import ARCH, CSRC, nvcc

SRC = """
#include "flags3d.cu"
#include "bisect.hpp"
#include "cluster2d.hpp"
using namespace amrb;
extern "C" int takes(int ndim, int is, int js, int ks, long long n) { return DeviceBisect::takes(ndim, LvlDims{is, js, ks}, (size_t)n); }
extern "C" int cut(const int* a, int na, const int* b, int nb, int* dir) {
  return find_cut_sig(std::vector<int>(a, a + na + 2), std::vector<int>(b, b + nb + 2), na, nb, *dir);
}
// the leaves of the tree (5 ints each: count, bounding box), or -1
extern "C" int leaves(const int* ij, int n, int is, int js, double cutoff, int max_nodes, long long max_wait, int* out, int room,
                      int* launched) {
  DeviceBisect bis;
  if (max_nodes > 0) bis.max_nodes = max_nodes;
  if (max_wait) bis.max_wait = max_wait;
  cudaStream_t st;
  if (cudaStreamCreate(&st) != cudaSuccess) return -2;
  int rc = -2;
  Staging stg;
  try {
    std::vector<unsigned long long> list(n);
    for (int k = 0; k < n; ++k) list[k] = bisect_point(ij[2 * k], ij[2 * k + 1], 1);
    std::vector<BisectNode> T;
    if (!bis.run(2, nullptr, LvlDims{is, js, 1}, list, cutoff, st, stg, T)) rc = -1;
    else {
      rc = 0;
      for (int id : DeviceBisect::leaves(T)) {
        if (rc == room) break;
        int* o = out + 5 * rc++;
        o[0] = T[id].n;
        for (int d = 0; d < 2; ++d) { o[1 + 2 * d] = T[id].clo[d]; o[2 + 2 * d] = T[id].chi[d]; }
      }
    }
    if (cudaStreamSynchronize(st) != cudaSuccess) rc = -3;
  } catch (std::exception& e) { std::fprintf(stderr, "%s\\n", e.what()); }
  *launched = bis.launched;
  bis.free(); stg.destroy(); cudaStreamDestroy(st);
  return rc;
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = str(tmp_path_factory.mktemp("bisect"))
    with open(d + "/bisect.cu", "w") as f:
        f.write(SRC)
    subprocess.run([nvcc(), "-std=c++17", "-O2", *ARCH, "--fmad=false", "-Xcompiler", "-fPIC", "-shared", "-I", CSRC, "-o",
                    d + "/bisect.so", d + "/bisect.cu"], check=True)
    return ctypes.CDLL(d + "/bisect.so")


def _p(a):
    return a.ctypes.data_as(ctypes.POINTER(ctypes.c_int))


def device(lib, pts, dims, cutoff, max_nodes=0, max_wait=0):
    pts = np.ascontiguousarray(pts, np.int32)
    out = np.zeros((20000, 5), np.int32)
    launched = ctypes.c_int()
    n = lib.leaves(_p(pts), len(pts), dims[0], dims[1], ctypes.c_double(cutoff), max_nodes, ctypes.c_longlong(max_wait), _p(out),
                   len(out), ctypes.byref(launched))
    return n if n < 0 else out[:n].tolist(), launched.value


def host(lib, pts, dims, cutoff):
    """smartbis.f over the host's findcut: the part at or above a cut first."""
    out, stack = [], [np.asarray(pts)]
    while stack:
        p = stack.pop()
        lo, hi = p.min(axis=0), p.max(axis=0)
        side = ctypes.c_int()
        c = 0
        if len(p) / float(int(hi[0] - lo[0] + 1) * int(hi[1] - lo[1] + 1)) < cutoff:
            sig = [np.bincount(p[:, d], minlength=dims[d] + 2).astype(np.int32) for d in (0, 1)]
            c = lib.cut(_p(sig[0]), dims[0], _p(sig[1]), dims[1], ctypes.byref(side))
        if c == 0:
            out.append([len(p), int(lo[0]), int(hi[0]), int(lo[1]), int(hi[1])])
            continue
        up = p[:, side.value - 1] >= c
        stack += [p[~up], p[up]]
    return out


def rectangles(boxes):
    pts = []
    for i0, i1, j0, j1 in boxes:
        i, j = np.meshgrid(np.arange(i0, i1 + 1), np.arange(j0, j1 + 1))
        pts.append(np.stack([i.ravel(), j.ravel()], axis=1))
    return np.unique(np.concatenate(pts), axis=0)


def outline(w, h, t):
    return rectangles([(3, 2 + t, 5, 4 + h), (3 + w - t, 2 + w, 5, 4 + h), (3, 2 + w, 5, 4 + t), (3, 2 + w, 5 + h - t, 4 + h)])


def test_levels_the_device_form_takes(lib):
    n = 1000
    assert lib.takes(2, 725, 725, 1, ctypes.c_longlong(n))       # one plane's cells are no limit in 2D
    assert lib.takes(2, 8192, 8192, 1, ctypes.c_longlong(n))
    assert lib.takes(2, 131072, 131072, 1, ctypes.c_longlong(2 << 20))
    assert not lib.takes(2, 131072, 131073, 1, ctypes.c_longlong(n))      # the counts of one node
    assert not lib.takes(2, 1024, 1024, 1, ctypes.c_longlong((2 << 20) + 1))
    assert lib.takes(3, 724, 724, 3, ctypes.c_longlong(0))
    assert not lib.takes(3, 725, 725, 2, ctypes.c_longlong(0))    # 2^19 points with one k


CASES = {
    "one point": (rectangles([(7, 7, 9, 9)]), (20, 20)),
    "two bands": (rectangles([(3, 6, 2, 40), (12, 30, 20, 22)]), (40, 44)),
    "past 725 squared": (outline(900, 900, 3), (1002, 1002)),
    "a box of 2^32 cells": (rectangles([(2, 9, 2, 9), (65530, 65537, 65530, 65537)]), (80000, 80000)),
    "47000 a line": (outline(29, 47000, 4), (40, 47100)),
    "65540 a line": (outline(29, 65540, 4), (40, 66000)),
}


@pytest.mark.gpu
@pytest.mark.parametrize("name", sorted(CASES))
@pytest.mark.parametrize("cutoff", [0.7, 0.97])
def test_trees(lib, name, cutoff):
    pts, dims = CASES[name]
    got, launched = device(lib, pts, dims, cutoff)
    assert launched == 2
    assert got == host(lib, pts, dims, cutoff)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1000, 8191, 8192, 140000])  # a block per 4096 points, at most 32
def test_scattered_points(lib, n):
    rng = np.random.default_rng(n)
    pts = np.unique(rng.normal((300, 500), (60, 90), (2 * n, 2)).astype(int).clip(1, 900), axis=0)
    pts = pts[rng.permutation(len(pts))[:n]]
    assert len(pts) > 0.1 * n
    got, _ = device(lib, pts, (1000, 1000), 0.6)
    assert got == host(lib, pts, (1000, 1000), 0.6)


@pytest.mark.gpu
def test_the_ways_out(lib):
    pts, dims = outline(3000, 3000, 3), (3200, 3200)
    assert len(pts) >= 8 * 4096  # several blocks, which wait for one another
    want = host(lib, pts, dims, 0.7)
    assert device(lib, pts, (131072, 131073), 0.7) == (-1, 0)
    assert device(lib, pts, dims, 0.7, max_nodes=3)[0] == -1
    assert device(lib, pts, dims, 0.7, max_wait=-1)[0] == -1  # every wait runs out at once
    assert device(lib, pts, dims, 0.7)[0] == want


@pytest.mark.gpu
def test_2d_run_past_the_device_limits(lib):
    """A level with more than 2^18 rows and columns: the waves decide, with signatures longer than
    a block's shared memory."""
    from amrclaw_b200 import Solver, problems
    from oracle.pyoracle import Oracle2D
    nx, ny = 20, 262200
    rd = problems.advection_square(8, 2, 2, 1.0, u=0.0, v=0.0, x0=5.0, x1=15.0, y0=100.0, y1=47100.0)
    c = rd.clawdata
    c.lower, c.upper, c.num_cells = [0.0, 0.0], [float(nx), float(ny)], [nx, ny]
    c.bc_lower = c.bc_upper = ["extrap", "extrap"]
    c.dt_initial = 0.1
    rd.amrdata.max1d = 2 * ny
    rd.amrdata.regrid_buffer_width = 1
    assert not lib.takes(2, nx, ny, 1, ctypes.c_longlong(1000))
    with tempfile.TemporaryDirectory() as d:
        rd.write(d)
        o = Oracle2D(d, threads=8)
        o.run(1)
        g, v = o.grids(), o.values()
        o.close()
        with Solver(d) as s:
            s.run(1)
            assert np.array_equal(s.grids(), g)
            assert np.array_equal(s.values(), v)
    assert (g[:, 1] == 2).sum() > 1
