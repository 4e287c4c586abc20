"""Cuts of clusters whose signatures jump by more than 46341 points: the product of the two
Laplacians there passes 32 bits, and the strongest cut must still be found. The flags are the
outline of a tall rectangle; its sides are then whole level-2 grids."""
import ctypes
import subprocess
import tempfile

import numpy as np
import pytest

import configs  # noqa: F401  (puts the repository on the path)
from amrclaw_b200 import problems
from amrclaw_b200.build import CSRC
from oracle.pyoracle import Oracle2D

H = 47000


def outline(nx, ny):
    rd = problems.advection_square(8, 2, 2, 1.0, u=0.0, v=0.0, x0=10.0, x1=nx - 10.0, y0=100.0, y1=100.0 + H)
    c = rd.clawdata
    c.lower, c.upper, c.num_cells = [0.0, 0.0], [float(nx), float(ny)], [nx, ny]
    c.bc_lower = c.bc_upper = ["extrap", "extrap"]
    c.dt_initial = 0.1
    rd.amrdata.max1d = 2 * ny
    rd.amrdata.regrid_buffer_width = 1
    return rd


def oracle_run(rd):
    with tempfile.TemporaryDirectory() as d:
        rd.write(d)
        o = Oracle2D(d, threads=8)
        o.run(1)
        g, v = o.grids(), o.values()
        o.close()
    return g, v


def test_oracle_cuts_off_the_tall_sides_first():
    g, _ = oracle_run(outline(40, H + 200))
    fine = g[g[:, 1] == 2]
    tall = fine[(fine[:, 5] - fine[:, 4] + 1) // 2 > H]
    assert len(fine) == 4 and len(tall) == 2
    assert (tall[:, 3] - tall[:, 2] + 1 < 20).all()


def test_host_cut_from_large_signatures():
    """find_cut_sig on the outline's signatures: the cut after the left band, not between the
    much weaker changes of the other direction."""
    src = '#include "cluster2d.hpp"\nextern "C" int cut(const int* a, int na, const int* b, int nb, int* dir) {' \
          "return amrb::find_cut_sig(std::vector<int>(a, a + na + 2), std::vector<int>(b, b + nb + 2), na, nb, *dir); }"
    with tempfile.TemporaryDirectory() as d:
        with open(d + "/cut.cpp", "w") as f:
            f.write(src)
        subprocess.run(["g++", "-O3", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, "-o", d + "/cut.so", d + "/cut.cpp"], check=True)
        lib = ctypes.CDLL(d + "/cut.so")
    for h in (50, 46338, 50000, 65532, 65536 + 4, 200000):
        i = np.zeros(30, np.int32)
        i[1:29] = 8
        i[1:5] = i[25:29] = h
        j = np.zeros(h + 2, np.int32)
        j[1:h + 1] = 8
        j[1:5] = j[h - 3:h + 1] = 28
        side = ctypes.c_int()
        p = lambda a: a.ctypes.data_as(ctypes.POINTER(ctypes.c_int))
        assert (lib.cut(p(i), 28, p(j), h, ctypes.byref(side)), side.value) == (5, 1), h


@pytest.mark.gpu
def test_device_hierarchy():
    from amrclaw_b200 import Solver
    rd = outline(40, H + 200)
    g, v = oracle_run(rd)
    with tempfile.TemporaryDirectory() as d:
        rd.write(d)
        with Solver(d) as s:
            s.run(1)
            assert np.array_equal(s.grids(), g)
            assert np.array_equal(s.values(), v)
