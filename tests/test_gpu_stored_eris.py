"""Stored ERIs of deeply contracted shells: a task's lanes share its quartets'
primitives (groups of 1 to 32 lanes), in classes from (ss|ss) to (dd|dd)."""
import time

import numpy as np
import pytest

from conftest import random_density
from iqcp_b200 import BasisSet, FockEngine
from iqcp_b200.molecules import REFERENCE_MOLECULES

pytestmark = pytest.mark.gpu
HCL = [(17, (0.1, -0.2, 0.3)), (1, (0.1, 0.4, 2.6))]


# 1 to 12 primitives a shell; absolute tolerance of the existing comparison with the
# oracle, per unit of the largest integral above 1 (36 for the tight shells of Cl)
@pytest.mark.parametrize("atoms,basis", [(HCL, "6-31g*"), (HCL, "cc-pvdz"), (HCL, "sto-3g"),
                                         (REFERENCE_MOLECULES["HF"], "6-31+g*")])
def test_blocks_against_the_oracle(oracle_mod, atoms, basis):
    b = BasisSet.build(atoms, basis)
    ref, _ = oracle_mod.eri_compressed(b)
    with FockEngine(b) as eng:
        out = eng.eri_compressed()
    assert np.abs(out - ref).max() <= 1e-13 * max(1.0, np.abs(ref).max())


def test_deep_contractions_do_not_wait_for_one_lane():
    """The same quartets as one J/K build, formed once: within ten times its duration.
    s and p shells only: the d blocks' own latency, up to 1296 components stored by a
    lane, is milliseconds whatever the contraction."""
    b = BasisSet.build(REFERENCE_MOLECULES["H2O"], "6-31g")
    D = random_density(b.n_basis, 1)

    def best(call):
        t = []
        for _ in range(7):
            t0 = time.perf_counter()
            call()
            t.append(time.perf_counter() - t0)
        return min(t)
    with FockEngine(b) as eng:
        assert best(eng.eri_compressed) < 10 * best(lambda: eng.build_jk(D))
