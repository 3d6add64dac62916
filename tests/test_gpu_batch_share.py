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


@pytest.mark.parametrize("config", [0, 2])
@pytest.mark.parametrize("plain", [0, 3000])    # 3000: the large ones as launches of their own
def test_every_instance_gets_its_own_tallies(plain, config):
    """Instances that differ in photons and media, on two meshes: the tallies of each one are
    those of a run by itself."""
    slab, abdomen = workloads.plain_slab(), workloads.curved_abdomen(freq=8)
    for w in (slab, abdomen):
        w.vox_n, w.n_rbins, w.det_r = (0, 0, 0), 0, None
        w.dimensions, w.det_grid = slab.dimensions, slab.det_grid
    rng = np.random.default_rng(2)
    inst = []
    for i, n in enumerate((1, 4000, 0, 33, 700, 5000, 2, 64, 3000, 90, 1, 250)):
        w = (slab, abdomen)[i % 2]
        media = np.array(w.nmuasg, np.float32)
        media[1:, 1:3] *= rng.uniform(0.8, 1.2, media[1:, 1:3].shape).astype(np.float32)
        inst.append(Instance(i % 2, media, n, 1000 * i))
    with slab.apply(Simulation(0), seed=3) as a, abdomen.apply(Simulation(0), seed=3) as c, Batch([a, c]) as b:
        b.set_plain_threshold(plain)
        b.set_config(config)
        b.set_instances(inst)
        b.run()
        for i, x in enumerate(inst):
            got, s = b.tallies(i), (a, c)[x.context]
            s.set_media(x.nmuasg)
            s.zero()
            s.run(x.n_photons, x.first)
            want = s.tallies()
            for key in ("sft", "rtd", "rz", "region"):
                assert np.array_equal(got[key], want[key]), (i, key)
            assert got["counters"]["photons"] == x.n_photons
