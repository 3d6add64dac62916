"""Contexts that are changed while a batch holds them: another mesh or cell grid is taken up by
the next run, another tally layout is refused (the batch's buffers are for the first)."""
import numpy as np
import pytest

from lightpropagation_b200 import Simulation, _native, workloads
from lightpropagation_b200.batch import Batch, Instance

pytestmark = pytest.mark.gpu

KEYS = ("sft", "rtd", "rz", "vox", "region")
N = 4000


def by_itself(w, cells, margin):
    with w.apply(Simulation(0), seed=3) as s:
        s.set_safety_grid(cells)
        s.set_cell_margin(margin)
        s.zero()
        s.run(N, 50)
        return s.tallies()


def same(b, want):
    got = b.tallies(0)
    for k in KEYS:
        assert np.array_equal(got[k], want[k]), k


@pytest.mark.parametrize("plain", [0, 1000])
@pytest.mark.parametrize("run_context", [False, True])
@pytest.mark.parametrize("set_again", [False, True])
def test_another_mesh_or_grid(plain, run_context, set_again):
    w, other = workloads.curved_abdomen(freq=8), workloads.curved_abdomen(freq=20, head_depth=50.0)
    inst = [Instance(0, w.nmuasg, N, 50), Instance(0, w.nmuasg, 0, 0)]
    with w.apply(Simulation(0), seed=3) as s, Batch([s]) as b:
        s.set_safety_grid(1 << 20)
        s.set_cell_margin(1.0)
        b.set_plain_threshold(plain)
        b.set_config(2)
        b.set_instances(inst)
        b.run()
        same(b, by_itself(w, 1 << 20, 1.0))
        for mesh, cells, margin in ((w, 1 << 20, 0.3), (w, 1 << 22, 0.5), (other, 1 << 22, 0.5), (w, 0, 0.5)):
            s.set_mesh(mesh.tri, mesh.nrm, mesh.med)
            s.set_safety_grid(cells)
            s.set_cell_margin(margin)
            if run_context:
                s.zero()
                s.run(100)
            if set_again:
                b.set_instances(inst)
            if run_context or set_again:     # the change has reached the device
                b.run()
                same(b, by_itself(mesh, cells, margin))


def test_another_layout_is_refused():
    w = workloads.plain_slab()
    with w.apply(Simulation(0), seed=3) as s, Batch([s]) as b:
        b.set_config(0)
        inst = [Instance(0, w.nmuasg, N, 50)]
        b.set_instances(inst)
        b.run()
        s.set_tally_grid(w.dimensions, np.asarray(w.det_grid) * np.float32(0.5), w.fetal_id)
        with pytest.raises(_native.LPError, match="tally layout"):
            b.set_instances(inst)
        s.set_tally_grid(w.dimensions, w.det_grid, w.fetal_id)
        b.set_instances(inst)
        b.run()
        assert b.tallies(0)["counters"]["photons"] == N
