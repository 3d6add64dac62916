"""The r-z deposits of a launch go to several copies of the image that are folded into the
tally afterwards; how many depends on the image's size and, in a batch, on the number of
instances.  Whatever the number, the tallies are the same integers."""
import numpy as np
import pytest

from lightpropagation_b200 import Simulation, workloads
from lightpropagation_b200.batch import Batch, Instance

pytestmark = pytest.mark.gpu


def configured(step, seed=17):
    """The slab with r and z bins of `step` mm: r-z images from 16 copies down to one."""
    w = workloads.plain_slab()
    w.det_grid = np.array([step, step, step, step, 1.0, 1.0], np.float32)
    return w.apply(Simulation(0), seed=seed)


# 0.1 MB (16 copies), 3.8 MB (8), 11 MB (2), 24 MB (1)
@pytest.mark.parametrize("step", [1.0, 0.16, 0.093, 0.063])
def test_rz_image_holds_every_deposit(step):
    """Every absorbed weight is in the r-z image exactly once: its sum is the regions'."""
    n = 3000
    with configured(step) as s:
        s.zero()
        s.run(n)
        one = s.tallies()
        s.zero()
        s.run(1000)
        s.run(n - 1000, 1000)
        two = s.tallies()
    assert one["counters"]["rz_drop"] == 0
    assert int(one["rz"][..., 0].sum()) == int(one["region"].sum()) > 0
    assert np.array_equal(one["rz"], two["rz"])


@pytest.mark.parametrize("plain", [0, 1])
def test_batch_rz_images_equal_single_runs(plain):
    """Instances of the shared launch (plain 0) and with a launch of their own (plain 1),
    each run twice: the copies are left at zero."""
    counts = [700, 1, 1500]
    with configured(1.0) as s:
        nm = workloads.plain_slab().nmuasg
        with Batch([s]) as b:
            b.set_plain_threshold(plain)
            b.set_instances([Instance(0, nm, n, 10 * i) for i, n in enumerate(counts)])
            b.run()
            b.run()
            got = [b.tallies(i)["rz"] for i in range(len(counts))]
        for i, n in enumerate(counts):
            s.zero()
            s.run(n, 10 * i)
            assert np.array_equal(s.tallies()["rz"], got[i]), i
