"""The sweeps of a 3D level on both sides of the size where its three directions stop sharing
one launch: bit-identical to the oracle."""
import tempfile

import numpy as np
import pytest

import configs
from oracle.pyoracle import Oracle3D

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells", [(4, 4, 4), (32, 32, 32), (32, 32, 36), (36, 34, 38)])
def test_levels_around_the_shared_launch(cells):
    from amrclaw_b200 import Solver
    rd = configs.euler_blast(n=32, levels=1, tfinal=1.0, max1d=60)
    rd.clawdata.num_cells = list(cells)
    rd.clawdata.dt_initial = 2e-3
    with tempfile.TemporaryDirectory() as d:
        rd.write(d)
        o = Oracle3D(d, threads=8)
        o.run(2)
        v = o.values()
        o.close()
        with Solver(d) as s:
            s.run(2)
            assert np.array_equal(s.values(), v)
