"""Nearest-triangle queries that march over the cell lists, against the BVH alone (which
test_gpu_parity compares with the full scan): the same id and the same bits of t at the
edges of the march."""
import numpy as np
import pytest

from lightpropagation_b200 import Simulation, meshes, workloads

pytestmark = pytest.mark.gpu


def rays(n, rng):
    """From inside, from outside (entering the grid or missing it), along the axes, on the
    grid's corner planes, with bounds from negative to beyond every hit."""
    o = rng.uniform(-160, 160, (n, 3))
    o[::5] *= 20.0
    d = rng.normal(size=(n, 3))
    d[1::4] = np.eye(3)[rng.integers(0, 3, len(d[1::4]))] * rng.choice([-1.0, 1.0], (len(d[1::4]), 1))
    d[::5] = rng.uniform(-100, 100, d[::5].shape) - o[::5]
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    t = rng.choice([-1.0, 0.0, 0.05, 0.7, 5.0, 60.0, 10000.0, 3e38], n)
    return o.astype(np.float32), d.astype(np.float32), np.full(n, -1, np.int32), t.astype(np.float32)


# margins of the lists (0: every march is stuck), cells of the grid (few: dense cells),
# counts around a warp and the queries it takes at a time
@pytest.mark.parametrize("margin,cells,n", [(0.5, 1 << 24, 20011), (0.0, 1 << 20, 3001), (2.0, 1 << 18, 3001),
                                            (0.5, 1 << 9, 3001), (0.5, 1 << 24, 1), (0.5, 1 << 24, 17),
                                            (0.5, 1 << 24, 33)])
def test_march_equals_bvh(margin, cells, n):
    tri, nrm, med = meshes.curved_abdomen(freq=14)
    q = rays(n, np.random.default_rng(5))
    got = []
    for lists in (False, True):
        with Simulation(0) as s:
            s.set_mesh(tri, nrm, med)
            s.set_safety_grid(cells)
            s.set_cell_margin(margin)
            s.set_cell_lists(lists)
            got.append(s.query(*q))
    assert np.array_equal(got[0][0], got[1][0])
    assert np.array_equal(got[0][1].view(np.uint32), got[1][1].view(np.uint32))
    if n > 1000:
        assert (got[0][0] >= 0).mean() > 0.1


@pytest.mark.parametrize("mesh", ["slab", "abdomen"])
@pytest.mark.parametrize("margin,cells", [(0.5, 1 << 24), (0.0, 1 << 20), (0.3, 1 << 16), (2.5, 1 << 20), (0.5, 1 << 6)])
def test_distance_bounds_change_no_tally(mesh, margin, cells):
    """The empty cells' distance bounds follow from the lists and their margin: with any
    margin and cell size, with and without the lists, the tallies are those of a run that
    queries every step."""
    w = workloads.plain_slab() if mesh == "slab" else workloads.curved_abdomen(freq=10)
    got = []
    for n_cells, lists in ((0, False), (cells, False), (cells, True)):
        with w.apply(Simulation(0), seed=77) as s:
            s.set_safety_grid(n_cells)
            s.set_cell_margin(margin)
            s.set_cell_lists(lists)
            s.zero()
            s.run(3000)
            got.append(s.tallies())
    for t in got[1:]:
        for k in ("sft", "rtd", "rz", "vox", "region"):
            assert np.array_equal(got[0][k], t[k]), k
