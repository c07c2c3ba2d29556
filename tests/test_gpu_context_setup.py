"""Contexts as a geometry scan makes them: task lists built on the device, memory
and streams handed from one context to the next, several host threads at once."""
import threading

import numpy as np
import pytest

from conftest import random_density
from iqcp_b200 import BasisSet, BatchFockEngine, FockEngine
from iqcp_b200.molecules import REFERENCE_MOLECULES, workload

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mol,basis", [("H2", "sto-3g"), ("H2O", "6-31+g*"), ("C6H6", "6-31g"), ("c1", "cc-pvdz")])
def test_all_quartets_without_screening(mol, basis):
    """Threshold 0 keeps every unique shell quartet (one class to six, up to
    several chunks of the task sum), each once."""
    atoms = workload("c1", 1)[0] if mol == "c1" else REFERENCE_MOLECULES[mol]
    b = BasisSet.build(atoms, basis)
    n = b.n_shells * (b.n_shells + 1) // 2
    D = random_density(b.n_basis, 1, 0.05)
    for thr in (0.0, 1e-12):
        with FockEngine(b, schwarz_threshold=thr) as eng:
            eng.build_jk(D)
            q = eng.last_stats()["quartets"]
            Q = eng.schwarz()
        pairs = np.sort(Q[np.tril_indices(b.n_shells)])
        # pairs (bra, ket) with bra >= ket and Q Q' >= thr, counted on the host
        both = sum(int((pairs * x >= thr).sum()) for x in pairs)
        assert q == (both + int((pairs * pairs >= thr).sum())) // 2
        assert thr > 0.0 or q == n * (n + 1) // 2


def test_batch_counts_are_the_sum():
    mols = [BasisSet.build(REFERENCE_MOLECULES[m], "6-31g*") for m in ("H2O", "CH4", "H2", "NH3")] * 3
    with BatchFockEngine(mols) as eng:
        eng.build_jk([random_density(b.n_basis, 2) for b in mols])
        total = eng.last_stats()["quartets"]
    one = 0
    for b in mols:
        with FockEngine(b) as eng:
            eng.build_jk(random_density(b.n_basis, 2))
            one += eng.last_stats()["quartets"]
    assert total == one


def test_many_contexts_from_threads():
    """Four threads make and destroy contexts that reuse each other's memory."""
    use = []
    for m in ("H2O", "CH4", "C6H6"):
        b = BasisSet.build(REFERENCE_MOLECULES[m], "6-31g*")
        D = random_density(b.n_basis, 3)
        with FockEngine(b) as eng:
            use.append((b, D) + tuple(eng.build_jk(D)) + (eng.eri_gradient(D),))
    bad = []

    def work(k):
        for i in range(6):
            b, D, J, K, g = use[(k + i) % len(use)]
            with FockEngine(b) as eng:
                Jt, Kt = eng.build_jk(D)
                gt = eng.eri_gradient(D)
            # the same sums in another atomic order
            if max(np.abs(Jt - J).max(), np.abs(Kt - K).max(), np.abs(gt - g).max()) > 1e-11:
                bad.append((k, i))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
