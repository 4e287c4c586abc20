"""The sweeps of a plugin without a quick form of its splits: one launch for the three directions
of a level of any size, identical to the oracle on grids of a few cells, of less than one wave of
tiles and of several."""
import tempfile

import numpy as np
import pytest

import configs
from oracle.pyoracle import Oracle3D

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells", [(4, 4, 4), (30, 32, 34), (52, 48, 50)])
def test_swirl_levels(cells):
    from amrclaw_b200 import Solver
    rd = configs.advection_swirl_regression()
    rd.clawdata.num_cells = list(cells)
    rd.clawdata.dt_initial = 2e-3
    rd.gaugedata.gauges = []
    rd.amrdata.amr_levels_max = 1
    rd.amrdata.max1d = 60
    with tempfile.TemporaryDirectory() as d:
        rd.write(d)
        o = Oracle3D(d, threads=8)
        o.run(2)
        v = o.values()
        o.close()
        with Solver(d) as s:
            s.run(2)
            assert np.array_equal(s.values(), v)
