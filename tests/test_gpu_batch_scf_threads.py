"""Batched SCFs and one-electron gradients of several host threads at once, one
context per thread: molecules whose kernels need different amounts of shared
memory must not change each other's launches, and contexts destroyed beside a
running SCF must not end its captures, nor be handed on while their own work
runs."""
import threading

import numpy as np
import pytest

from conftest import random_density
from iqcp_b200 import BasisSet, BatchFockEngine, FockEngine
from iqcp_b200.batch_scf import BatchRHF
from iqcp_b200.molecules import REFERENCE_MOLECULES

pytestmark = pytest.mark.gpu


def _in_threads(works):
    errors, start = [], threading.Barrier(len(works))

    def guarded(work):
        try:
            start.wait(60)
            work()
        except Exception as e:  # reported by the main thread
            errors.append(repr(e))
    threads = [threading.Thread(target=guarded, args=(w,)) for w in works]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[0]


@pytest.mark.parametrize("pair", [(("C6H6", "6-31g*"), ("C6H6", "cc-pvdz")),   # 102 and 120 functions
                                  (("C6H6", "6-31g"), ("CH4", "cc-pvdz"))])    # 66 and 35: two forms of the step
def test_two_batched_scfs(pair):
    """Two SCFs whose purification steps share a kernel (or not) converge as they
    do alone: to the 1e-9 Ha and 1e-7 of their own thresholds."""
    bases = [BasisSet.build(REFERENCE_MOLECULES[m], b) for m, b in pair]
    alone = []
    for b in bases:
        scf = BatchRHF([b])
        res = scf.run()
        alone.append((res.energies[0], scf.densities()[0]))
        scf.close()
    got = [[], []]

    def run(k):
        scf = BatchRHF([bases[k]])
        for _ in range(4):
            res = scf.run()
            got[k].append((bool(res.converged.all()), res.energies[0], scf.densities()[0]))
        scf.close()
    _in_threads([lambda: run(0), lambda: run(1)])
    for k in range(2):
        assert len(got[k]) == 4
        for ok, e, D in got[k]:
            assert ok and abs(e - alone[k][0]) < 1e-9 and np.abs(D - alone[k][1]).max() < 1e-6


def test_two_one_electron_gradients_of_many_atoms():
    """Launches of 1400 and 2000 atoms hold 34 and 48 KB of gradient in shared
    memory; both agree with the single molecule (sums of a few terms: 1e-13)."""
    b = BasisSet.build(REFERENCE_MOLECULES["H2"], "sto-3g")
    rng = np.random.default_rng(2)
    D = rng.normal(size=(2, 2))
    W = rng.normal(size=(2, 2))
    D, W = D + D.T, W + W.T
    with BatchFockEngine([b]) as eng:
        ref = eng.one_electron_gradient([D], [W])[0]
    bad = []

    def run(n):
        with BatchFockEngine([b] * n) as eng:
            for _ in range(20):
                g = eng.one_electron_gradient([D] * n, [W] * n)
                if max(np.abs(x - ref).max() for x in g) > 1e-13:
                    bad.append(n)
    _in_threads([lambda: run(700), lambda: run(1000)])
    assert not bad


def test_contexts_destroyed_beside_a_batched_scf():
    """A batched SCF captures an iteration; threads that make and destroy contexts
    meanwhile leave the capture alone (errors of a capture ended by another
    thread come back as a failed SCF)."""
    b = BasisSet.build(REFERENCE_MOLECULES["NH3"], "6-31g*")
    small = BasisSet.build(REFERENCE_MOLECULES["H2"], "sto-3g")
    scf = BatchRHF([b])
    e0 = scf.run().energies[0]
    D = random_density(2, 1)
    with FockEngine(small) as eng:
        J0, K0 = eng.build_jk(D)
    left = [12]
    bad = []

    def iterate():
        try:
            while left[0] > 0:
                res = scf.run()
                left[0] -= 1
                if not res.converged.all() or abs(res.energies[0] - e0) > 1e-9:
                    bad.append(res.energies[0])
        finally:
            left[0] = 0

    def churn():
        while left[0] > 0:
            with FockEngine(small) as eng:
                J, K = eng.build_jk(D)
            if max(np.abs(J - J0).max(), np.abs(K - K0).max()) > 1e-12:
                bad.append("J/K")
    _in_threads([iterate, churn, churn])
    scf.close()
    assert not bad, bad


@pytest.mark.parametrize("captured", [False, True])
def test_destroy_waits_for_enqueued_work(captured):
    """A context destroyed right after a call that only enqueues (or the replay of a
    graph that captured one) on the caller's stream, and the next context in its
    memory: the first call's results are those of a call waited for (1e-12)."""
    import torch
    b = BasisSet.build(REFERENCE_MOLECULES["CH4"], "6-31g*")
    n = b.n_basis
    D1, D2 = random_density(n, 1, 0.05), random_density(n, 2, 0.05)
    with FockEngine(b) as eng:
        ref = eng.build_jk(D1)
    stream = torch.cuda.Stream()
    d = torch.from_numpy(D1).cuda()
    J, K = torch.zeros_like(d), torch.zeros_like(d)
    for _ in range(4):
        eng = FockEngine(b)
        eng.set_stream(stream.cuda_stream)
        eng.jk_device_noalloc(d.data_ptr(), J.data_ptr(), K.data_ptr())
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        if captured:
            with torch.cuda.graph(graph, stream=stream):
                eng.jk_device_noalloc(d.data_ptr(), J.data_ptr(), K.data_ptr())
        J.zero_()
        K.zero_()
        torch.cuda.synchronize()
        with torch.cuda.stream(stream):
            torch.cuda._sleep(20_000_000)
            if captured:
                graph.replay()
            else:
                eng.jk_device_noalloc(d.data_ptr(), J.data_ptr(), K.data_ptr())
        eng.close()
        with FockEngine(b) as other:   # on streams and memory of the first
            other.build_jk(D2)
        torch.cuda.synchronize()
        del graph
        assert np.abs(J.cpu().numpy() - ref[0]).max() < 1e-12
        assert np.abs(K.cpu().numpy() - ref[1]).max() < 1e-12
