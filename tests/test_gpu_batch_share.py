"""How the warps of the batch launch share out its instances: uneven budgets, empty and
one-photon instances, more instances than a warp looks at at once, totals below and above
the lanes of the launch.  Every instance is traced once, whole."""
import numpy as np
import pytest

from lightpropagation_b200 import Simulation, workloads
from lightpropagation_b200.batch import Batch, Instance

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("config", [0, 2])
@pytest.mark.parametrize("counts", [(0, 1, 0), (5000,), (1, 20000, 0, 3, 700), tuple(range(0, 75))])
def test_every_instance_is_traced_once(counts, config):
    w = workloads.plain_slab()
    with w.apply(Simulation(0), seed=3) as s:
        with Batch([s]) as b:
            b.set_plain_threshold(0)
            b.set_config(config)
            # the same total twice (the graph is kept), then another one
            for first, scale in ((0, 1), (9, 1), (0, 2)):
                n = [scale * c for c in counts]
                b.set_instances([Instance(0, w.nmuasg, c, first) for c in n])
                b.run()
                got = [b.tallies(i) for i in range(len(n))]
                assert [t["counters"]["photons"] for t in got] == n
                k = int(np.argmax(n))
                s.zero()
                s.run(n[k], first)
                want = s.tallies()
                for key in ("sft", "rz", "vox", "rbins"):
                    assert np.array_equal(got[k][key], want[key]), key
