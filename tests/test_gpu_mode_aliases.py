"""The kernel variants that exist: modes 2 and 3 are accepted and run mode 0, tuning
picks only modes with kernels of their own, and FP64 classes of more than 108
components are the warp kernels' alone.  Sums in another atomic order: 1e-11."""
import numpy as np
import pytest

from conftest import random_density
from iqcp_b200 import MIXED, BasisSet, FockEngine
from iqcp_b200.molecules import REFERENCE_MOLECULES

pytestmark = pytest.mark.gpu
COMPS = [1, 3, 9, 6, 18, 36]


@pytest.mark.parametrize("mode", [2, 3])
def test_modes_2_and_3_are_mode_0(mode):
    b = BasisSet.build(REFERENCE_MOLECULES["NH3"], "6-31g*")
    D = random_density(b.n_basis, 4, 0.1)
    out = []
    with FockEngine(b) as eng:
        for m in (0, mode):
            eng.set_kernel_mode("jk", mode=m)
            eng.set_kernel_mode("grad", mode=m)
            out.append(tuple(eng.build_jk(D)) + (eng.eri_gradient(D),))
    for x, y in zip(*out):
        assert np.abs(x - y).max() < 1e-11


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_tuning_picks_kernels_that_exist(precision):
    import torch
    b = BasisSet.build(REFERENCE_MOLECULES["C6H6"], "6-31g*")   # all 21 classes
    D = random_density(b.n_basis, 5, 0.1)
    with FockEngine(b) as eng:
        if precision == "mixed":
            eng.set_precision(MIXED, 1e-3)
        modes = eng.autotune(torch.from_numpy(D).cuda().data_ptr(), 1)
    for X in range(6):
        for Y in range(6):
            for kind in range(4):
                m = modes[kind, X, Y]
                if Y > X:
                    assert m == -1
                elif kind < 2:
                    assert m == 1 if COMPS[X] * COMPS[Y] > 108 else m in (0, 1)
                else:
                    assert m in (0, 1, 4)
