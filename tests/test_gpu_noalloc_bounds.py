"""lp_run_noalloc skips the queries that the distance to the mesh rules out, found over the
whole mesh (small ones) or its tree: the tallies stay those of lp_run in reference
arithmetic, on either side of that size, for open meshes and for scenes of another scale or
far from the origin."""
import ctypes as C

import numpy as np
import pytest

from lightpropagation_b200 import _native, workloads
from test_zz_no_alloc import KEYS, _args, regular

pytestmark = pytest.mark.gpu


def cut(n_tri, scale, shift):
    """The first n_tri triangles of a coarse abdomen, scaled and moved along x."""
    w = workloads.curved_abdomen(freq=2)
    t = np.array([shift, 0.0, 0.0], np.float32)
    w.tri = (w.tri[:n_tri].reshape(-1, 3) * np.float32(scale) + t).reshape(-1, 9).astype(np.float32)
    w.nrm, w.med = w.nrm[:n_tri], w.med[:n_tri]
    w.p_start = (w.p_start * np.float32(scale) + t).astype(np.float32)
    w.ep0xyz = w.ep0xyz.copy()
    w.ep0xyz[:3] = w.ep0xyz[:3] * np.float32(scale) + t
    w.dimensions = (w.dimensions * np.float32(scale)).astype(np.float32)
    w.det_grid = w.det_grid.copy()
    w.det_grid[:4] *= np.float32(scale)
    w.nmuasg = w.nmuasg.copy()
    w.nmuasg[:, 1:3] /= np.float32(scale)
    w.vox_n, w.n_rbins, w.det_r = (0, 0, 0), 0, None
    w.fiber_radius *= scale
    return w


@pytest.mark.parametrize("n_tri,scale,shift", [(1, 1.0, 0.0), (31, 1.0, 0.0), (33, 1.0, 0.0), (256, 1.0, 0.0),
                                               (257, 1.0, 0.0), (400, 1.0, 0.0), (256, 40.0, 0.0), (400, 0.05, 0.0),
                                               (256, 1.0, 900.0), (400, 1.0, 900.0)])
def test_bounds_change_no_tally(n_tri, scale, shift):
    import torch

    w = cut(n_tri, scale, shift)
    n, seed = 3000, 17
    ref, g = regular(w, n, seed)
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


@pytest.mark.parametrize("mesh", ["slab", "abdomen"])
def test_many_photons_change_no_tally(mesh):
    """Above 64 photons for each of 16 warps per SM (151,552 on 148 SMs) the kernel's other
    instance runs, with more blocks and fewer registers."""
    import torch

    dev = torch.device("cuda", 0)
    n, seed = 64 * 16 * torch.cuda.get_device_properties(dev).multi_processor_count + 4099, 29
    w = workloads.plain_slab() if mesh == "slab" else workloads.curved_abdomen(freq=3)
    ref, g = regular(w, n, seed)
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
