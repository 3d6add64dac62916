"""A batch whose lp_batch_set_instances runs out of memory (injected on the host): it has no
instances then, and takes new ones as if nothing had happened."""
import numpy as np
import pytest

from lightpropagation_b200 import Simulation, _native, workloads
from lightpropagation_b200.batch import Batch, Instance

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("plain", [0, 1000])    # 1000: the second kind of buffers too
def test_no_instances_until_the_next_ones(plain):
    L = _native.lib()
    w = workloads.plain_slab()
    n = 1500
    with w.apply(Simulation(0), seed=6) as s:
        s.zero()
        s.run(n, 2 * n)
        want = s.tallies()
        failures = 0
        try:
            for k in range(40):
                with Batch([s]) as b:
                    b.set_plain_threshold(plain)
                    b.set_config(0)
                    b.set_instances([Instance(0, w.nmuasg, n, i * n) for i in range(2)])
                    b.run()
                    L.lp_debug_fail_allocation(k)
                    try:
                        b.set_instances([Instance(0, w.nmuasg, n, i * n) for i in range(20)])
                        failed = False
                    except _native.LPError:
                        failed = True
                    L.lp_debug_fail_allocation(-1)
                    if failed:
                        failures += 1
                        b.run()                      # nothing to trace
                        with pytest.raises(_native.LPError):
                            b.tallies(0)
                        b.set_instances([Instance(0, w.nmuasg, n, i * n) for i in range(3)])
                    b.run()
                    got = b.tallies(2)
                    for key in ("sft", "rz", "vox", "region"):
                        assert np.array_equal(got[key], want[key]), (k, key)
                if not failed:
                    break
        finally:
            L.lp_debug_fail_allocation(-1)
        assert failures >= 10, failures
