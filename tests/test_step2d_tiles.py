"""The 2D patch step against the oracle at the edges of its tiles: grids smaller than a tile,
one cell short of it and past it, several tiles with ragged remainders, for every plugin that
needs no aux, with and without the second-order and the transverse terms. The quadrant
problem has subsonic and supersonic interfaces, in both directions. Bit-identical."""
import tempfile

import numpy as np
import pytest

from amrclaw_b200 import problems
from oracle.pyoracle import Oracle2D

pytestmark = pytest.mark.gpu

BUILD = {"advection": lambda: problems.advection_square(16, 1, 2, 1.0),
         "acoustics": lambda: problems.acoustics_pulse(16, 1, 2, 1.0),
         "euler": lambda: problems.euler_quadrants(16, 1, 2, 1.0, xs=0.6, ys=0.55)}


@pytest.mark.parametrize("kind", sorted(BUILD))
@pytest.mark.parametrize("cells,levels", [((4, 6), 1), ((14, 16), 1), ((16, 18), 1), ((18, 34), 2), ((50, 30), 2)])
@pytest.mark.parametrize("order,trans", [(2, 2), (2, 1), (2, 0), (1, 1), (1, 0)])
def test_tiles_identical_to_the_oracle(kind, cells, levels, order, trans):
    from amrclaw_b200 import Solver
    rd = BUILD[kind]()
    c, a = rd.clawdata, rd.amrdata
    c.num_cells = list(cells)
    c.order, c.transverse_waves = order, trans
    c.dt_initial = 0.05 / max(cells)
    c.cfl_desired = 0.9 if order == 2 and trans == 2 else 0.4
    a.amr_levels_max = levels
    with tempfile.TemporaryDirectory() as d:
        rd.write(d)
        o = Oracle2D(d, threads=4)
        o.run(5)
        g, v, t = o.grids(), o.values(), o.time()
        o.close()
        with Solver(d) as s:
            s.run(5)
            assert np.array_equal(s.grids(), g)
            assert s.info()["time"] == t
            w = s.values()
    assert np.isfinite(v).all()
    assert np.array_equal(w, v)
