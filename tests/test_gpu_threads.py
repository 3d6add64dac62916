"""Contexts of several threads that stage different amounts of shared memory, and a captured
launch between calls that do: the limit of dynamic shared memory is the kernel's, not a call's."""
import ctypes as C
import threading

import numpy as np
import pytest

from lightpropagation_b200 import Simulation, _native, workloads
from test_zz_no_alloc import KEYS, _args, regular

pytestmark = pytest.mark.gpu


def test_threads_with_different_budgets():
    slab, abdomen = workloads.plain_slab(), workloads.curved_abdomen(freq=10)
    jobs = [(slab, 8, False), (abdomen, 8, False), (abdomen, 120, False), (abdomen, 40, True), (slab, 8, True),
            (abdomen, 200, True)]

    def trace(job, times):
        w, kb, exact = job
        out = []
        with w.apply(Simulation(0), seed=5) as s:
            s.set_smem_budget(kb * 1024)
            s.set_arithmetic(exact)
            for k in range(times):
                s.zero()
                s.run(500 + 100 * k)
                t = s.tallies()
                out.append([np.array(t[key]) for key in ("sft", "rz", "region")])
                s.query(w.p_start[None], w.v_start[None])
        return out

    want = [trace(j, 8) for j in jobs]
    got, errors = [None] * len(jobs), []

    def work(i):
        try:
            got[i] = trace(jobs[i], 8)
        except Exception as e:   # reported by the test's thread
            errors.append((jobs[i][1:], e))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(jobs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for a, b in zip(got, want):
        for x, y in zip(a, b):
            assert all(np.array_equal(p, q) for p, q in zip(x, y))


@pytest.mark.parametrize("mesh", ["slab", "abdomen"])
def test_captured_noalloc_between_other_calls(mesh):
    """lp_run_noalloc in a CUDA graph: replayed after calls that stage less and more, the
    tallies are those of lp_run each time."""
    import torch

    w = workloads.plain_slab() if mesh == "slab" else workloads.curved_abdomen(freq=4)
    other = workloads.curved_abdomen(freq=4) if mesh == "slab" else workloads.plain_slab()
    n, seed = 2000, 13
    ref, g = regular(w, n, seed)
    dev = torch.device("cuda", 0)

    def call_of(w, n):
        tri, nrm, med = (torch.from_numpy(np.ascontiguousarray(x, t).ravel()).to(dev)
                         for x, t in ((w.tri, np.float32), (w.nrm, np.float32), (w.med, np.int32)))
        nm = np.ascontiguousarray(w.nmuasg, np.float32).ravel()
        geo = regular(w, 1, seed)[1]
        sizes = {"sft": geo.sft_nx * geo.sft_ny * 3, "rtd": geo.dimR * geo.dimAlpha * 3,
                 "rz": geo.rz_nr * geo.rz_nz * 2, "region": w.nmuasg.shape[0], "counters": 16}
        out = {k: torch.zeros(v, dtype=torch.int64, device=dev) for k, v in sizes.items()}
        a = _args(w, seed, n, tri, nrm, med, nm, out)
        return a, out, (tri, nrm, med, nm)

    L = _native.lib()
    a, out, keep = call_of(w, n)
    b, _, keep_b = call_of(other, 100)
    stream = torch.cuda.Stream(dev)
    with torch.cuda.stream(stream):
        assert L.lp_run_noalloc(C.byref(a), C.c_void_p(stream.cuda_stream)) == 0   # outside of a capture first
    stream.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        for t in out.values():
            t.zero_()
        assert L.lp_run_noalloc(C.byref(a), C.c_void_p(stream.cuda_stream)) == 0
    for _ in range(3):
        assert L.lp_run_noalloc(C.byref(b), C.c_void_p(torch.cuda.current_stream(dev).cuda_stream)) == 0
        torch.cuda.synchronize(dev)
        graph.replay()
        torch.cuda.synchronize(dev)
        for k in KEYS:
            assert np.array_equal(out[k].cpu().numpy().view(np.uint64), ref[k].ravel()), k
