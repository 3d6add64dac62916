"""Runs of a few photons: how many share a warp decides how their random numbers are drawn
(each lane its own, or several events ahead for the photons that are left), and no number
of them changes a tally."""
import numpy as np
import pytest

from lightpropagation_b200 import Simulation, workloads

pytestmark = pytest.mark.gpu

KEYS = ("sft", "rtd", "rz", "vox", "rbins", "region")


@pytest.mark.parametrize("exact", [False, True])
def test_photons_in_one_run_equal_photons_one_by_one(exact):
    # 1 photon, edges of the groups of 2, 4, 8, 16 and 32 lanes, more than a warp
    counts = (1, 2, 3, 4, 5, 8, 9, 16, 17, 32, 33, 70)
    with workloads.plain_slab().apply(Simulation(0), seed=23) as s:
        s.set_arithmetic(exact)
        s.zero()
        for n in range(max(counts) + 1):
            if n in counts:
                one_by_one = s.tallies()
                with workloads.plain_slab().apply(Simulation(0), seed=23) as t:
                    t.set_arithmetic(exact)
                    t.zero()
                    t.run(n)
                    together = t.tallies()
                for k in KEYS:
                    assert np.array_equal(one_by_one[k], together[k]), (n, k)
                assert one_by_one["counters"]["scatter"] == together["counters"]["scatter"], n
            s.run(1, n)
