"""The 3D Euler transverse splits against the oracle where their forms change over: tiles that
are subsonic throughout, tiles with supersonic interfaces (a strong blast drives the gas
faster than its sound speed), and the tiny numerators of the fluctuations ahead of a front.
FP64 results are bit-identical whichever form a tile takes."""
import tempfile

import numpy as np
import pytest

import configs
from oracle.pyoracle import Oracle3D

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gamma,pin,r0,cfl,n,max1d,supersonic", [
    (1.4, 1.0001, 0.2, 0.9, 14, 18, False), (1.4, 5.0, 0.2, 0.9, 18, 12, None), (1.1, 100.0, 0.2, 0.3, 16, 20, True),
    (1.2, 300.0, 0.35, 0.3, 22, 26, True)])
def test_splits_identical_to_the_oracle(gamma, pin, r0, cfl, n, max1d, supersonic):
    from amrclaw_b200 import Solver
    rd = configs.euler_blast(n=n, levels=2, tfinal=1.0, max1d=max1d)
    for k, v in (("gamma", gamma), ("pin", pin), ("r0", r0)):
        rd.probdata.add_param(k, v)
    rd.clawdata.dt_initial = float(0.02 / n / np.sqrt(pin))
    rd.clawdata.cfl_desired = cfl
    with tempfile.TemporaryDirectory() as d:
        rd.write(d)
        o = Oracle3D(d, threads=8)
        o.run(16)
        g, v, t = o.grids(), o.values(), o.time()
        o.close()
        with Solver(d) as s:
            s.run(16)
            assert np.array_equal(s.grids(), g)
            assert s.info()["time"] == t
            w = s.values()
    assert np.isfinite(v).all()
    assert np.array_equal(w, v)
    if supersonic is not None:  # the base level is one grid
        q = v[:5 * n ** 3].reshape(5, -1)
        p = (gamma - 1.0) * (q[4] - 0.5 * (q[1] ** 2 + q[2] ** 2 + q[3] ** 2) / q[0])
        mach = np.abs(q[1:4]).max(axis=0) / q[0] / np.sqrt(gamma * p / q[0])
        assert (mach.max() > 1.0) == supersonic
