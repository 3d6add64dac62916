"""A CUDA call that fails is reported by the entry point that made it, and by no later one."""
import numpy as np
import pytest

from lightpropagation_b200 import Simulation, _native, workloads

pytestmark = pytest.mark.gpu


def test_a_failed_allocation_fails_no_later_launch():
    L = _native.lib()
    one = np.zeros(1, np.float32)
    w = workloads.plain_slab()
    with w.apply(Simulation(0), seed=2) as s:
        s.zero()
        s.run(500)
        want = s.tallies()
    for again in (0, 1):
        # 4 TiB, refused by cudaMalloc before the arrays are looked at
        assert L.lp_exact_ops(0, 0, 1 << 40, _native.fptr(one), _native.fptr(one), _native.fptr(one)) == 4
        assert b"memory" in L.lp_last_error(None)
        with w.apply(Simulation(0), seed=2) as s:
            s.zero()
            s.run(500)
            got = s.tallies()
        assert np.array_equal(got["sft"], want["sft"]) and np.array_equal(got["rz"], want["rz"])
