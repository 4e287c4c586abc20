"""2D boundary ops against the oracle: walls, extrapolation and periodic sides mixed, corners
between them, grids as narrow as their ghost regions, coarse scratch arrays of refined levels
at the boundary. Bit-identical."""
import tempfile

import numpy as np
import pytest

from amrclaw_b200 import problems
from oracle.pyoracle import Oracle2D

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells,levels", [((2, 2), 1), ((4, 30), 1), ((24, 20), 3)])
@pytest.mark.parametrize("lower,upper", [(("wall", "wall"), ("wall", "wall")), (("wall", "extrap"), ("extrap", "wall")),
                                         (("periodic", "wall"), ("periodic", "extrap")),
                                         (("extrap", "periodic"), ("wall", "periodic"))])
def test_boundaries_identical_to_the_oracle(cells, levels, lower, upper):
    from amrclaw_b200 import Solver
    rd = problems.acoustics_pulse(20, levels, 2, 1.0, r0=0.9, width=0.3)
    c = rd.clawdata
    c.num_cells = list(cells)
    c.bc_lower, c.bc_upper = list(lower), list(upper)
    c.dt_initial = 0.02 / max(cells)
    c.cfl_desired = 0.45
    with tempfile.TemporaryDirectory() as d:
        rd.write(d)
        o = Oracle2D(d, threads=4)
        o.run(6)
        g, v = o.grids(), o.values()
        o.close()
        with Solver(d) as s:
            s.run(6)
            assert np.array_equal(s.grids(), g)
            w = s.values()
    assert np.isfinite(v).all()
    assert np.array_equal(w, v)
