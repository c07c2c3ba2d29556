"""Which classes of a mixed call run an FP32 share before autotuning: those of
more than 108 components, or the largest where none is.  Forced to FP64, every
class gives the FP64 results.

Tolerances: FP64 against FP64 in another order of atomic additions, 1e5 of
them at 1e-16 each, 1e-11 relative to the largest element; FP32 quadrature of
every quartet of the split classes, 2e-5 as in the variants' own test."""
import numpy as np
import pytest

from conftest import random_density
from iqcp_b200 import MIXED, BasisSet, FockEngine
from iqcp_b200.molecules import REFERENCE_MOLECULES

pytestmark = pytest.mark.gpu

COMPS = [1, 3, 9, 6, 18, 36]  # ss, ps, pp, ds, dp, dd


@pytest.mark.parametrize("mol,basis,least", [("H2", "6-31g", 1), ("C6H6", "6-31g", 81), ("C6H6", "6-31g*", 109)])
def test_default_split(mol, basis, least):
    b = BasisSet.build(REFERENCE_MOLECULES[mol], basis)
    D = random_density(b.n_basis, 7, 0.2)
    with FockEngine(b) as eng:
        ref = (*eng.build_jk(D), eng.eri_gradient(D, 1.0))
        eng.set_precision(MIXED, 1e30)
        modes = eng.kernel_modes()
        for X in range(6):
            for Y in range(X + 1):
                if modes[0, X, Y] >= 0:
                    assert ((modes[2:, X, Y] != 4) == (COMPS[X] * COMPS[Y] >= least)).all()
        out = []
        for kind in ("default", "fp64"):
            if kind == "fp64":
                eng.set_kernel_mode("jk32", mode=4)
                eng.set_kernel_mode("grad32", mode=4)
            J, K = eng.build_jk(D)
            n = eng.last_stats()["fp32_quartets"]
            g = eng.eri_gradient(D, 1.0)
            assert (n > 0) == (eng.last_stats()["fp32_quartets"] > 0) == (kind == "default")
            out.append((J, K, g))
    for x, mixed, fp64 in zip(ref, *out):
        assert np.abs(mixed - x).max() <= 2e-5 * np.abs(x).max()
        assert np.abs(fp64 - x).max() <= 1e-11 * np.abs(x).max()
