"""What a mesh keeps on the device: 64 bytes a tree node, 48 a triangle and 16 for its
attributes, and nothing of its upload."""
import pytest

from lightpropagation_b200 import Simulation, workloads

pytestmark = pytest.mark.gpu


def test_mesh_keeps_nothing_of_its_upload():
    import torch

    small, large = workloads.curved_abdomen(freq=4), workloads.curved_abdomen(freq=80)
    with small.apply(Simulation(0), seed=1) as s:
        s.set_safety_grid(0)
        s.run(0)
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info(0)[0]
        s.set_mesh(large.tri, large.nrm, large.med)
        s.run(0)
        torch.cuda.synchronize()
        kept = before - torch.cuda.mem_get_info(0)[0]
        nodes = s.stats()["n_nodes"]
    # six buffers in blocks of 2 MiB; a copy of the triangles would be 30 MB more
    assert kept <= 64 * nodes + 64 * large.n_tri + 6 * (2 << 20), (kept, nodes, large.n_tri)
