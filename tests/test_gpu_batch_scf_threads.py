"""Batched SCFs and one-electron gradients of several host threads at once, one
context per thread: molecules whose kernels need different amounts of shared
memory must not change each other's launches."""
import threading

import numpy as np
import pytest

from iqcp_b200 import BasisSet, BatchFockEngine
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
