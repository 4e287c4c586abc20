"""Clusters of the one-launch bisection against the oracle's hierarchies: point lists for one
block and for several (a wide band of flags), and a level past the device form's limits,
which the host bisects wave by wave."""
import tempfile

import numpy as np
import pytest

import configs
from amrclaw_b200 import problems
from oracle.pyoracle import Oracle2D, Oracle3D

pytestmark = pytest.mark.gpu


def _same(rd, oracle, steps):
    from amrclaw_b200 import Solver
    with tempfile.TemporaryDirectory() as d:
        rd.write(d)
        o = oracle(d, threads=8)
        o.run(steps)
        g, v = o.grids(), o.values()
        o.close()
        with Solver(d) as s:
            s.run(steps)
            assert np.array_equal(s.grids(), g)
            assert np.array_equal(s.values(), v)
    return g


@pytest.mark.parametrize("n,tol,cutoff", [(40, 0.2, 0.7), (40, 0.05, 0.95), (200, 1e-3, 0.8), (300, 1e-4, 0.6)])
def test_2d_hierarchies(n, tol, cutoff):
    rd = problems.acoustics_pulse(n, 2, 2, 1.0)
    rd.amrdata.flag2refine_tol = tol
    rd.amrdata.clustering_cutoff = cutoff
    g = _same(rd, Oracle2D, 5)
    assert (g[:, 1] == 2).any()


@pytest.mark.parametrize("cutoff", [0.5, 0.9])
def test_3d_hierarchies(cutoff):
    rd = configs.euler_blast(n=24, levels=3, tfinal=1.0, max1d=20)
    rd.amrdata.clustering_cutoff = cutoff
    g = _same(rd, Oracle3D, 3)
    assert (g[:, 1] == 3).any()


def test_3d_level_past_the_device_limits():
    rd = configs.euler_blast(n=4, levels=2, tfinal=1.0, max1d=2000)
    rd.clawdata.num_cells = [1024, 514, 2]  # more than 2^19 cells in a plane
    rd.probdata.add_param("z0", -0.5)
    rd.clawdata.dt_initial = 1e-4
    g = _same(rd, Oracle3D, 1)
    assert (g[:, 1] == 2).any()
