"""Reference arithmetic where its divisions by optical constants and bin widths take one or
the other path (correctly rounded by multiplication, or the operator): photons follow the
oracle's as in the parity tests (over nine tenths of the exit records to 1e-4)."""
import numpy as np
import pytest

import pyoracle as po
from conftest import to_case
from lightpropagation_b200 import Simulation, workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,mua,mus,g,step", [
    ("usual", 0.02, 2.0, 0.9, 1.0),
    ("isotropic", 0.02, 2.0, 0.0, 1.0),
    ("backward", 0.02, 2.0, -0.7, 0.37),
    ("g below the range", 0.02, 2.0, 1e-7, 1.0),
    ("g above the range", 0.02, 2.0, 0.9999998, 1.0),
    ("mua below the range", 1e-13, 2.0, 0.9, 1.0),
])
def test_exit_records_follow_the_oracle(oracle_lib, name, mua, mus, g, step):
    w = workloads.plain_slab()
    w.nmuasg = w.nmuasg.copy()
    w.nmuasg[1:, 1], w.nmuasg[1:, 2], w.nmuasg[1:, 3] = mua, mus, g
    w.det_grid = np.array([1.0, 1.0, step, 0.5 * step, 1.0, 1.0], np.float32)
    n, seed = 400, 31
    with w.apply(Simulation(0), seed=seed) as s:
        s.set_arithmetic(True)
        s.set_exit_records(n)
        s.zero()
        s.run(n)
        rec, t = s.exit_records(n), s.tallies()
    r = po.run(to_case(w), n, rng_mode=po.RNG_PHILOX, seed=seed, exit_records=True)
    close = np.all(np.isclose(rec, r.exit_rec, rtol=1e-4, atol=1e-5), axis=1).mean()
    assert close > 0.9, close
    assert t["counters"]["photons"] == n
