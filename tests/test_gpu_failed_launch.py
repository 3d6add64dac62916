"""Launches that fail (injected on the host by lp_debug_fail_launch): the deposits in the copies
of the r-z image neither get lost nor turn up in a later result."""
import numpy as np
import pytest

from lightpropagation_b200 import Simulation, _native, workloads
from lightpropagation_b200.batch import Batch, Instance

pytestmark = pytest.mark.gpu

KEYS = ("sft", "rtd", "rz", "vox", "region")
N = 3000


@pytest.fixture
def fail_launch():
    L = _native.lib()
    yield L.lp_debug_fail_launch
    L.lp_debug_fail_launch(-1)


def equal(got, want):
    for k in KEYS:
        assert np.array_equal(got[k], want[k]), k


def clean(runs):
    with workloads.plain_slab().apply(Simulation(0), seed=4) as s:
        s.zero()
        for n, first in [(0, 0)] + runs:     # 0 photons: the tallies exist
            s.run(n, first)
        return s.tallies()


@pytest.mark.parametrize("which", [0, 1])   # the transport launch, the fold of its deposits
@pytest.mark.parametrize("then", ["zero", "read", "run on", "restore"])
def test_context(fail_launch, which, then):
    with workloads.plain_slab().apply(Simulation(0), seed=4) as s:
        s.zero()
        s.run(N, 7 * N)
        saved = s.checkpoint()
        s.zero()
        fail_launch(which)
        with pytest.raises(_native.LPError):
            s.run(N)
        fail_launch(-1)
        done = [(N, 0)] if which else []     # the photons that were traced all the same
        if then == "zero":
            s.zero()
            s.run(N, 5 * N)
            equal(s.tallies(), clean([(N, 5 * N)]))
        elif then == "read":
            equal(s.tallies(), clean(done))
        elif then == "run on":
            s.run(N, 2 * N)
            equal(s.tallies(), clean(done + [(N, 2 * N)]))
        else:
            s.restore(saved)
            s.run(N, 3 * N)
            equal(s.tallies(), clean([(N, 7 * N), (N, 3 * N)]))


@pytest.mark.parametrize("which", [0, 1, 3, 5])   # a launch of the autotuner's, a fold of its
def test_batch(fail_launch, which):
    w = workloads.plain_slab()
    with w.apply(Simulation(0), seed=4) as s, Batch([s]) as b:
        b.set_plain_threshold(0)
        # 60 photons at which every step counts, so the autotuner's launches have as many
        inst = [Instance(0, w.nmuasg, 32, 0), Instance(0, w.nmuasg, 28, 32)]
        b.set_instances(inst)
        fail_launch(which)
        with pytest.raises(_native.LPError):
            b.autotune()
        fail_launch(-1)
        b.set_instances(inst)
        b.set_config(0)
        b.run()
        equal(b.tallies(0), clean([(32, 0)]))
        equal(b.tallies(1), clean([(28, 32)]))


@pytest.mark.parametrize("which", [0, 1, 4])
def test_autotuner_puts_the_budgets_back(fail_launch, which):
    w = workloads.plain_slab()
    with w.apply(Simulation(0), seed=4) as s, Batch([s]) as b:
        b.set_plain_threshold(0)
        b.set_instances([Instance(0, w.nmuasg, N, 0), Instance(0, w.nmuasg, 2 * N, N)])
        fail_launch(which)
        with pytest.raises(_native.LPError, match="launch"):
            b.autotune(64)
        fail_launch(-1)
        b.set_config(0)
        b.run()
        equal(b.tallies(0), clean([(N, 0)]))
        equal(b.tallies(1), clean([(2 * N, N)]))
