"""The workloads whose run time this repository watches.

Each case is one pass through the public entry points as a user's program makes it, on
the repository's own workloads (``lightpropagation_b200.workloads``): the planar slab of
the plain method, the curved abdomen at its two wavelengths and the deformed abdomen.
The optical properties and the Philox seed come from the case's seed; the mesh is the
case's.

A pass returns the fixed-point tallies (integers), the counters of physical events and,
where the entry point has them, the ring signals, derivatives, images and exit records.
The counters that say how the library answered its mesh queries (executed, skipped,
through the tree) describe the implementation and are left out.
"""
import ctypes
import functools
import math

import numpy as np
import torch

from lightpropagation_b200 import Simulation, _native, workloads
from lightpropagation_b200.batch import Batch, Instance
from lightpropagation_b200.diff import ring_signals
from lightpropagation_b200.propagation import CalculatePropagation

EVENTS = ("scatter", "boundary", "roulette", "miss", "capped", "rz_drop", "vox_drop", "photons", "region_mismatch")
TALLIES = ("sft", "rtd", "rz", "vox", "rbins", "region", "det")

# scattering events per photon of each mesh's workload (counted by the library), for work()
EVENTS_PER_PHOTON = {"slab": 2580, "abdomen": 1350, "deformed": 1350}
# FP32 operations of one event: random numbers, step, direction update, deposits
FLOPS_PER_EVENT = 64


def listed():
    return [
        # a quick look at a new setting: a thousand photons, where the call's own latency counts
        {"name": "slab_1k", "entry": "run", "mesh": "slab", "freq": 0, "wavelength": 660, "photons": 1000},
        # the plain method at its stated photon count
        {"name": "slab_1m", "entry": "run", "mesh": "slab", "freq": 0, "wavelength": 660, "photons": 1_000_000},
        # verification against the reference: its order of operations, with exit records
        {"name": "slab_exact_100k", "entry": "exact", "mesh": "slab", "freq": 0, "wavelength": 660, "photons": 100_003},
        # one of many short runs on the abdomen (a scan over optical properties), an odd count
        {"name": "abdomen660_100k", "entry": "run", "mesh": "abdomen", "freq": 45, "wavelength": 660, "photons": 99_991},
        # the curved abdomen at its default count
        {"name": "abdomen660_10m", "entry": "run", "mesh": "abdomen", "freq": 45, "wavelength": 660,
         "photons": 10_000_000},
        # one step of a fit through torch: ring signals and the gradient of a loss on them
        {"name": "abdomen940_autograd_1m", "entry": "autograd", "mesh": "abdomen", "freq": 45, "wavelength": 940,
         "photons": 1_000_000},
        # the seven-region displaced mesh
        {"name": "deformed940_500k", "entry": "run", "mesh": "deformed", "freq": 45, "wavelength": 940,
         "photons": 500_000},
        # the drop-in launcher on a new model each time (25,600 triangles, as the largest
        # shipped model): setters, Init, Propagation, images
        {"name": "launcher_new_model_50k", "entry": "launcher", "mesh": "abdomen", "freq": 16, "wavelength": 660,
         "photons": 50_000},
        # the batched forward workload, small budgets: instances with uneven photon counts
        # on three meshes at both wavelengths, ring signals out
        {"name": "batch_forward_32", "entry": "batch", "mesh": "abdomen", "freq": 30, "wavelength": 660,
         "photons": 1_000_000, "instances": 32},
        # one step of the inverse loop: new absorptions, one differentiated batch
        {"name": "batch_fit_step_8", "entry": "batch_fit", "mesh": "deformed", "freq": 45, "wavelength": 660,
         "photons": 400_000, "instances": 8},
        # a caller whose device memory is its own: the transport without allocation
        {"name": "noalloc_slab_50k", "entry": "noalloc", "mesh": "slab", "freq": 0, "wavelength": 660,
         "photons": 50_000},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    entry = rng.choice(["run", "run", "run", "exact", "autograd", "launcher", "batch", "batch_fit", "noalloc"])
    mesh = rng.choice(["slab", "abdomen", "abdomen", "deformed"])
    if entry in ("autograd", "batch", "batch_fit") and mesh == "slab":
        mesh = "abdomen"
    most = {"run": 4_000_000, "exact": 400_000, "autograd": 1_500_000, "launcher": 300_000, "batch": 2_000_000,
            "batch_fit": 1_000_000, "noalloc": 100_000}[entry]
    freq = 0 if mesh == "slab" else rng.randint(6, 48)
    if entry == "noalloc":
        # within the entry point's 4096 triangles
        mesh, freq = ("slab", 0) if mesh == "slab" else ("abdomen", rng.randint(4, 6))
    case = {"entry": entry, "mesh": mesh, "freq": freq, "wavelength": rng.choice([660, 940]),
            "photons": _log(rng, 500 if entry != "batch" else 20_000, most) | 1}
    if entry in ("batch", "batch_fit"):
        case["instances"] = rng.randint(2, 40)
    return case


@functools.lru_cache(maxsize=8)
def _workload(mesh, freq, wavelength, head_depth=40.0):
    if mesh == "slab":
        return workloads.plain_slab()
    if mesh == "abdomen":
        return workloads.curved_abdomen(wavelength=wavelength, freq=freq, head_depth=head_depth)
    return workloads.deformed_abdomen(wavelength=wavelength, freq=freq)


def _media(w, rng):
    """The workload's optical properties within a few percent, one draw per region."""
    t = np.array(w.nmuasg, np.float32)
    t[1:, 1:3] *= rng.uniform(0.95, 1.05, t[1:, 1:3].shape).astype(np.float32)
    return t


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    w = _workload(case["mesh"], case["freq"], case["wavelength"])
    entry, n = case["entry"], case["photons"]
    key = int(rng.integers(1, 1 << 62))
    s = {"entry": entry, "n": n, "w": w}
    if entry == "launcher":
        media = _media(w, rng)
        c = CalculatePropagation()
        c.SetSeed(key)
        c.SetCompat(w.compat)
        s.update(launcher=c, media=media)
        return s
    if entry == "noalloc":
        return _prepare_noalloc(s, w, n, _media(w, rng), key)
    if entry in ("batch", "batch_fit"):
        return _prepare_batch(s, case, w, rng, key)
    sim = w.apply(Simulation(0), seed=key)
    media = _media(w, rng)
    sim.set_media(media)
    s["sim"] = sim
    if entry == "exact":
        sim.set_arithmetic(True)
        sim.set_exit_records(n)
    if entry == "autograd":
        s["media"] = media
        s["mua"] = torch.from_numpy(media[:, 1].copy()).double().requires_grad_()
        s["mus"] = torch.from_numpy(media[:, 2].copy()).double().requires_grad_()
        s["weight"] = torch.from_numpy(rng.uniform(0.5, 2.0, len(w.det_r)))
    return s


def _prepare_batch(s, case, w, rng, key):
    k, n = case["instances"], case["photons"]
    if case["entry"] == "batch":
        meshes = [w] + [_workload(case["mesh"], max(6, case["freq"] - 6), 660, depth) for depth in (47.5, 61.0)]
    else:
        meshes = [w]
    s["sims"] = [m.apply(Simulation(0), seed=key) for m in meshes]
    s["batch"] = Batch(s["sims"])
    # log-uniform budgets over a factor of ten, scaled to the case's total
    share = np.exp(rng.uniform(0.0, math.log(10.0), k)) if case["entry"] == "batch" else np.ones(k)
    budget = np.maximum((share / share.sum() * n).astype(np.int64), 32)
    first, inst = 0, []
    for i in range(k):
        wave = 660 if i % 2 == 0 else 940
        bf, sp = rng.uniform(0.02, 0.08, 2), rng.uniform(0.3, 0.7)
        table = workloads.tissue_table(wave, rng.uniform(0.9, 1.0), sp, bf[0], bf[1], np.exp(0.05 * rng.standard_normal(6)))
        if len(w.nmuasg) > len(table):
            table = np.vstack([table, w.nmuasg[len(table):]])
        inst.append(Instance(context=i % len(meshes), nmuasg=table, n_photons=int(budget[i]), first=first))
        first += int(budget[i])
    s["instances"] = inst
    if case["entry"] == "batch":
        s["batch"].set_instances(inst)
    else:
        s["batch"].set_gradient(True)
    return s


def _prepare_noalloc(s, w, n, media, key):
    dev = torch.device("cuda", 0)
    s["mesh"] = [torch.from_numpy(np.ascontiguousarray(x, t).ravel()).to(dev)
                 for x, t in ((w.tri, np.float32), (w.nrm, np.float32), (w.med, np.int32))]
    s["media"] = np.ascontiguousarray(media, np.float32).ravel()
    nx, ny, nz = (int(w.dimensions[i] / w.det_grid[i]) for i in range(3))
    n_alpha = int(90 / w.det_grid[5])
    n_r = math.ceil(math.hypot(nx // 2, ny // 2))
    sizes = {"sft": (2 * (nx // 2) + 1) * (2 * (ny // 2) + 1) * 3, "rtd": n_r * n_alpha * 3,
             "rz": (2 * n_r + 1) * (nz + 1) * 2, "region": len(media), "counters": _native.NCOUNTERS}
    s["out"] = {k: torch.zeros(v, dtype=torch.int64, device=dev) for k, v in sizes.items()}
    a = _native.NoAllocArgs()
    a.tri, a.nrm, a.med, a.n_tri = *(t.data_ptr() for t in s["mesh"]), w.n_tri
    a.nmuasg, a.n_media = _native.fptr(s["media"]), len(media)
    a.p_start[:] = [float(x) for x in w.p_start]
    a.v_start[:] = [float(x) for x in w.v_start]
    a.ep0xyz[:] = [float(x) for x in w.ep0xyz]
    a.fiber_radius = w.fiber_radius
    a.fiber_cos_max = w.src_cos_max if (w.fiber_radius > 0 or w.fiber_na > 0) else 1.0
    a.dimensions[:] = [float(x) for x in w.dimensions]
    a.det_grid[:] = [float(x) for x in w.det_grid]
    a.fetal_id, a.chance, a.w_threshold, a.factor = w.fetal_id, w.chance, w.w_threshold, w.factor
    a.seed, a.compat, a.first, a.n_photons = key, w.compat, 0, n
    a.sft, a.rtd, a.rz = (s["out"][k].data_ptr() for k in ("sft", "rtd", "rz"))
    a.region, a.counters = s["out"]["region"].data_ptr(), s["out"]["counters"].data_ptr()
    s["args"] = a
    return s


def _integers(t):
    out = {k: t[k].view(np.int64) for k in TALLIES}
    out["events"] = np.array([t["counters"][k] for k in EVENTS], np.int64)
    return out


def run(s):
    entry, n = s["entry"], s["n"]
    if entry in ("run", "exact"):
        sim = s["sim"]
        sim.zero()
        sim.run(n)
        out = _integers(sim.tallies())
        if entry == "exact":
            out["exit"] = sim.exit_records(n)
        return out
    if entry == "autograd":
        s["mua"].grad = s["mus"].grad = None
        signal = ring_signals(s["sim"], s["media"], s["mua"], s["mus"], n)
        (signal * s["weight"]).sum().backward()
        return {"signal": signal.detach(), "mua": s["mua"].grad, "mus": s["mus"].grad}
    if entry == "launcher":
        return _run_launcher(s)
    if entry == "batch":
        s["batch"].run()
        signal, err = s["batch"].ring_signals()
        return {"signal": signal, "error": err}
    if entry == "batch_fit":
        b = s["batch"]
        b.set_instances(s["instances"])
        b.run()
        g = [b.gradient(i) for i in range(len(s["instances"]))]
        return {k: np.stack([x[k] for x in g]) for k in ("signal", "signal_se", "d_mua", "d_mus")}
    for t in s["out"].values():
        t.zero_()
    stream = torch.cuda.current_stream().cuda_stream
    rc = _native.lib().lp_run_noalloc(ctypes.byref(s["args"]), ctypes.c_void_p(stream))
    _native.check(rc)
    out = dict(s["out"])
    # scatter, boundary, roulette, miss, capped, photons: the physical events
    out["counters"] = s["out"]["counters"][[0, 1, 3, 4, 5, 8]]
    return out


def _run_launcher(s):
    w, c = s["w"], s["launcher"]
    m = s["media"]
    c.SetTriangles(w.tri)
    c.SetNormals(w.nrm)
    c.SetInnerAndOuterTissueIndices(w.med)
    c.SetTissueProperties(m[:, 0], m[:, 1], m[:, 3], m[:, 2])
    c.SetStartPoint(w.p_start)
    c.SetStartTrajectories(w.v_start, [1])
    c.eP0XYZ = [float(x) for x in w.ep0xyz]
    c.SetDimensions(w.dimensions)
    c.SetDetectionGridDimensions(w.det_grid)
    c.SetFetalTissueID(w.fetal_id)
    c.SetChanceForRoulette(w.chance)
    c.SetWeightThreshold(w.w_threshold)
    c.SetPixelPerUnitFactor(w.factor)
    c.SetNumberOfPhotons(s["n"])
    c.Init()
    c.Propagation()
    out = _integers(c.GetTallies())
    out["sft_image"], out["rtd_image"] = c.GetSFTImage().data, c.GetRTdImage().data
    out["rz_image"], out["phi_image"] = c.GetArzImage().data, c.GetPhirzImage().data
    return out


def work(case):
    """Bytes: mesh and optical properties read once, the tallies written once.  Operations:
    the events of the photon paths."""
    w = _workload(case["mesh"], case["freq"], case["wavelength"])
    k = case.get("instances", 1)
    nx, ny, nz = (int(w.dimensions[i] / w.det_grid[i]) for i in range(3))
    n_r = math.ceil(math.hypot(nx // 2, ny // 2))
    cells = 3 * (nx + 1) * (ny + 1) + 3 * n_r * int(90 / w.det_grid[5]) + 2 * (2 * n_r + 1) * (nz + 1)
    if case["entry"] not in ("launcher", "noalloc"):
        cells += math.prod(w.vox_n) + 2 * w.n_rbins
    events = case["photons"] * EVENTS_PER_PHOTON[case["mesh"]]
    return {"bytes": 56 * w.n_tri + 16 * k * len(w.nmuasg) + 8 * k * cells, "flops": FLOPS_PER_EVENT * events}


def exact(case, seed):
    """None: the integer tallies are held bit for bit, and the floating outputs are ratios
    of sums over the same photon paths.  A path branches on single-precision comparisons
    thousands of times, so a 64-bit trace of the same photon is another path and gives a
    sample of the same distribution, not the value that these outputs approximate."""
    return None
