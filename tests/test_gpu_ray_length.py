"""Directions of any length: a ray's t counts in units of its direction, as in the reference
(MCLightPropagation.cl:1037-1093), whichever way the query is answered."""
import ctypes as C

import numpy as np
import pytest

from lightpropagation_b200 import Simulation, _native, meshes, workloads
from test_zz_no_alloc import KEYS, _args

pytestmark = pytest.mark.gpu


# a little beyond the rounding of a unit direction, far beyond it, and shorter ones
@pytest.mark.parametrize("length", [0.1, 0.99, 1.00001, 1.5, 2.0, 50.0])
@pytest.mark.parametrize("mesh", ["slab", "abdomen"])
def test_query_takes_directions_of_any_length(mesh, length):
    """The cell lists against the tree alone: the same triangles and the same bits of t, for
    bounds from a fraction of a cell to the default, in which the ray's hits lie."""
    tri, nrm, med = meshes.curved_abdomen(freq=14) if mesh == "abdomen" else (
        lambda w: (w.tri, w.nrm, w.med))(workloads.plain_slab())
    rng = np.random.default_rng(8)
    n = 6007
    lo, hi = tri.reshape(-1, 3).min(0), tri.reshape(-1, 3).max(0)
    o = rng.uniform(lo - 0.2 * (hi - lo), hi + 0.2 * (hi - lo), (n, 3))
    d = rng.normal(size=(n, 3))
    d *= length / np.linalg.norm(d, axis=1, keepdims=True)
    t = rng.choice([0.05, 0.7, 5.0, 30.0, 10000.0], n) / length
    q = (o.astype(np.float32), d.astype(np.float32), np.full(n, -1, np.int32), t.astype(np.float32))
    got = []
    for lists in (False, True):
        with Simulation(0) as s:
            s.set_mesh(tri, nrm, med)
            s.set_cell_lists(lists)
            got.append(s.query(*q))
    assert np.array_equal(got[0][0], got[1][0])
    assert np.array_equal(got[0][1].view(np.uint32), got[1][1].view(np.uint32))
    assert (got[0][0] >= 0).sum() > 300   # enough hits to compare


def beam(mesh, length, exterior):
    """A pencil beam of the workload whose direction has the given length, from air or from a
    scattering medium around the mesh."""
    w = workloads.plain_slab() if mesh == "slab" else workloads.curved_abdomen(freq=10)
    w.fiber_radius = w.fiber_na = 0.0
    w.v_start = (np.asarray(w.v_start, np.float32) * np.float32(length)).astype(np.float32)
    w.nmuasg = w.nmuasg.copy()
    if exterior == "scattering":
        w.nmuasg[0, 1:] = 0.01, 0.5, 0.8
    return w


@pytest.mark.parametrize("length", [0.3, 1.5, 20.0])
@pytest.mark.parametrize("exterior", ["air", "scattering"])
@pytest.mark.parametrize("mesh", ["slab", "abdomen"])
@pytest.mark.parametrize("exact", [False, True])
def test_run_takes_a_source_direction_of_any_length(mesh, exterior, length, exact):
    """The first step goes along the source's direction as given: the tallies of a run with
    the cell grid are those of a run that descends the tree on every step."""
    w = beam(mesh, length, exterior)
    got = []
    for cells in (0, 1 << 22):
        with w.apply(Simulation(0), seed=21) as s:
            s.set_arithmetic(exact)
            s.set_safety_grid(cells)
            s.zero()
            s.run(3000)
            got.append(s.tallies())
    for k in ("sft", "rtd", "rz", "vox", "region"):
        assert np.array_equal(got[0][k], got[1][k]), k
    c = got[0]["counters"]
    assert c["scatter"] + c["boundary"] >= 3000   # from air, only a direction of unit length gets in


@pytest.mark.parametrize("length", [0.3, 1.5, 20.0])
@pytest.mark.parametrize("exterior", ["air", "scattering"])
@pytest.mark.parametrize("mesh", ["slab", "abdomen"])
def test_noalloc_takes_a_source_direction_of_any_length(mesh, exterior, length):
    """lp_run_noalloc with such a beam, on either side of the mesh size up to which a query
    goes through the whole mesh, gives the tallies of lp_run without the cell grid."""
    import torch

    w = beam(mesh, length, exterior)
    w.tri, w.nrm, w.med = w.tri[:_native.NOALLOC_MAX_TRI], w.nrm[:_native.NOALLOC_MAX_TRI], w.med[:_native.NOALLOC_MAX_TRI]
    n, seed = 3000, 23
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
    for k in KEYS:
        assert np.array_equal(out[k].cpu().numpy().view(np.uint64), ref[k].ravel()), k
    cnt = out["counters"].cpu().numpy()
    assert int(cnt[8]) == n and int(cnt[0]) == ref["counters"]["scatter"]
