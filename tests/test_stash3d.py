"""Levels whose pencils do not fit the sweeps' staging memory in whole groups of eight slots lie
packed there: grids of two cells a side, on which the groups would take 2.7 times the memory,
on both paths. Identical to the oracle."""
import tempfile

import numpy as np
import pytest

import configs
from oracle.pyoracle import Oracle3D

pytestmark = pytest.mark.gpu

N = 24


def slots(grids, pad):
    """Slots of a level's pencils, each rounded up to whole groups of pad + 1."""
    n = [grids[:, 2 * d + 3] - grids[:, 2 * d + 2] + 1 for d in range(3)]
    return sum(int(((n[(d + 1) % 3] + 2) * (n[(d + 2) % 3] + 2) * ((n[d] + 1 + pad) & ~pad)).sum()) for d in range(3))


@pytest.mark.parametrize("batched", [True, False])
def test_grids_of_two_cells(batched):
    from amrclaw_b200 import Solver
    rd = configs.euler_blast(n=N, levels=2, tfinal=1.0, max1d=6)
    with tempfile.TemporaryDirectory() as d:
        rd.write(d)
        o = Oracle3D(d, threads=8)
        o.run(3)
        g, v = o.grids(), o.values()
        o.close()
        with Solver(d, batched=batched) as s:
            s.run(3)
            assert np.array_equal(s.grids(), g)
            assert np.array_equal(s.values(), v)
    base = g[g[:, 1] == 1]
    room = 2 * max(slots(base, 0), 3 * (N ** 3 + 12 * N * N))  # what the stash grows to for it
    assert slots(base, 7) > room
