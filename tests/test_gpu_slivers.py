"""Meshes of slivers (aspect ratios of some hundreds to a million): the rounding of a
triangle's own geometry must not turn into a distance bound that is too large, or a cell
list that is too short."""
import ctypes as C

import numpy as np
import pytest

from lightpropagation_b200 import Simulation, _native, meshes, workloads
from test_zz_no_alloc import KEYS, _args

pytestmark = pytest.mark.gpu


def fans(w, parts, turn):
    """The slab with each triangle of its four planes cut into a fan of `parts` slivers, whose
    vertices are then turned (which of them is the reference vertex of the hit test)."""
    tri, med = [], []
    for t, m in zip(w.tri.reshape(-1, 3, 3).astype(np.float64), w.med):
        k = parts if np.ptp(t[:, 2]) == 0.0 else 1
        edge = t[1] + (t[2] - t[1]) * (np.arange(k + 1) / k)[:, None]
        for i in range(k):
            tri.append(np.roll(np.stack([t[0], edge[i], edge[i + 1]]), turn, axis=0))
            med.append(m)
    w.tri = np.asarray(tri, np.float32).reshape(-1, 9)
    w.nrm, w.med = meshes.face_normals(w.tri), np.asarray(med, np.int32)
    return w


@pytest.mark.parametrize("turn", [0, 1, 2])
@pytest.mark.parametrize("parts", [40, 160, 500])
def test_noalloc_bounds_on_slivers(parts, turn):
    """lp_run_noalloc, whose bounds are distances to the triangles, gives the tallies of lp_run
    without a grid, which descends the tree on every step."""
    import torch

    w = fans(workloads.plain_slab(), parts, turn)
    w.nmuasg = w.nmuasg.copy()
    w.nmuasg[1:, 2] = 4.0, 0.4, 1.0     # steps of up to the layers' size
    assert 256 < w.n_tri <= _native.NOALLOC_MAX_TRI
    n, seed = 10000, 61
    with w.apply(Simulation(0), seed=seed) as s:
        s.set_arithmetic(True)
        s.set_safety_grid(0)
        s.zero()
        s.run(n)
        ref, g = s.tallies(), s.geometry()
    dev = torch.device("cuda", 0)
    tri, nrm, med = (torch.from_numpy(np.ascontiguousarray(x, t).ravel()).to(dev)
                     for x, t in ((w.tri, np.float32), (w.nrm, np.float32), (w.med, np.int32)))
    nm = np.ascontiguousarray(w.nmuasg, np.float32).ravel()
    sizes = {"sft": g.sft_nx * g.sft_ny * 3, "rtd": g.dimR * g.dimAlpha * 3, "rz": g.rz_nr * g.rz_nz * 2,
             "region": w.nmuasg.shape[0], "counters": 16}
    out = {k: torch.zeros(v, dtype=torch.int64, device=dev) for k, v in sizes.items()}
    a = _args(w, seed, n, tri, nrm, med, nm, out)
    rc = _native.lib().lp_run_noalloc(C.byref(a), C.c_void_p(torch.cuda.current_stream(dev).cuda_stream))
    assert rc == 0
    torch.cuda.synchronize(dev)
    cnt = out["counters"].cpu().numpy()
    for k in KEYS:
        assert np.array_equal(out[k].cpu().numpy().view(np.uint64), ref[k].ravel()), k
    assert int(cnt[8]) == n and int(cnt[0]) == ref["counters"]["scatter"]


@pytest.mark.parametrize("aspect", [1e3, 1e5, 1e6])
def test_cell_lists_hold_slivers(aspect):
    """Needles in every direction and rays aimed at them: the lists' triangles and bits of t are
    the tree's, with a margin and without one that neighbouring cells would make up for.  (From
    1e7 on a width is a unit or two of the coordinates, and the hit test itself, as the
    reference has it, can put a hit millimetres off the needle, where no list looks for it.)"""
    rng = np.random.default_rng(3)
    n = 3000
    a = rng.uniform(-60, 60, (n, 3))
    e, f = rng.normal(size=(2, n, 3))
    e *= rng.uniform(10, 80, (n, 1)) / np.linalg.norm(e, axis=1, keepdims=True)
    f *= np.linalg.norm(e, axis=1, keepdims=True) / aspect / np.linalg.norm(f, axis=1, keepdims=True)
    tri = np.stack([a, a + e, a + rng.uniform(0, 1, (n, 1)) * e + f], 1).astype(np.float32)
    nrm = np.tile(np.array([0, 0, 1], np.float32), (n, 1))
    med = np.tile(np.array([1, 0], np.int32), (n, 1))
    k = rng.integers(0, n, 40000)
    u = rng.uniform(0, 1, (len(k), 2))
    u = np.where(u.sum(1, keepdims=True) > 1, 1 - u, u)
    t = tri.astype(np.float64)[k]
    x = t[:, 0] + u[:, :1] * (t[:, 1] - t[:, 0]) + u[:, 1:] * (t[:, 2] - t[:, 0])
    d = rng.normal(size=x.shape)
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    o = (x - d * rng.choice([0.3, 3.0, 30.0], (len(k), 1))).astype(np.float32)
    q = (o, d.astype(np.float32), np.full(len(k), -1, np.int32),
         rng.choice([0.4, 4.0, 40.0, 10000.0], len(k)).astype(np.float32))
    for margin in (0.0, 0.5):
        got = []
        for lists in (False, True):
            with Simulation(0) as s:
                s.set_mesh(tri.reshape(-1, 9), nrm, med)
                s.set_cell_margin(margin)
                s.set_cell_lists(lists)
                got.append(s.query(*q))
        assert np.array_equal(got[0][0], got[1][0]), margin
        assert np.array_equal(got[0][1].view(np.uint32), got[1][1].view(np.uint32)), margin
