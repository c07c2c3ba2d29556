"""The Hermite gradient kernel (ss and ps kets) at the sizes where it changes:
T = 0 and both sides of the Boys table's end, more bra primitives than a warp
stages at a time, and the Rys kernels (mode 1, a warp per quartet) on the
same quartets.

Tolerance: every term is formed to a few ulp and the sums cancel by translation
invariance at most to the size of the largest derivative; 1e-10 relative to it
allows for the horizontal transfer of the Rys side (see test_gpu_lane_groups)."""
import numpy as np
import pytest

from conftest import random_density
from iqcp_b200 import BasisSet, FockEngine

pytestmark = pytest.mark.gpu


def basis(ls, n, xyz, lo=0.25, hi=40.0):
    rng = np.random.default_rng(len(ls) + n)
    xyz = np.asarray(xyz, float)
    at = np.repeat(np.arange(len(xyz)), len(ls))
    ex = np.geomspace(lo, hi, n) if n > 1 else np.array([0.8])
    return BasisSet("h", [2] * len(xyz), xyz, list(ls) * len(xyz), [n] * len(at), at, xyz[at], ex.tolist() * len(at),
                    rng.uniform(0.1, 0.4, n * len(at)))


CASES = {
    # all on one centre: T = 0 everywhere
    "one centre": ((0, 1, 2), 2, [[0.2, -0.1, 0.4]]),
    # exponents 0.8: T = 0.8 R^2 crosses 36 between the centres (6.7 bohr)
    "table end": ((0, 1, 2), 1, [[0, 0, 0], [0, 0.1, 6.6], [0.05, 0, 6.8], [0.3, 0.2, 14.0]]),
    # 16 to 49 bra primitives: several stages of p and d bras
    "staged bra": ((1, 2), 4, [[0, 0, 0], [1.1, 0.3, -0.4]]),
    "deep s and p": ((0, 1), 7, [[0, 0, 0], [0.9, -0.7, 0.5]]),
}


@pytest.mark.parametrize("name", list(CASES))
def test_against_oracle_and_rys(oracle_mod, name):
    b = basis(*CASES[name])
    D = random_density(b.n_basis, 3)
    oracle_mod.set_root_precision(True)
    try:
        go, _ = oracle_mod.eri_gradient(b, D, 0.7)
    finally:
        oracle_mod.set_root_precision(False)
    out = []
    with FockEngine(b) as eng:
        for mode in (0, 1):
            eng.set_kernel_mode("grad", mode=mode)
            out.append(eng.eri_gradient(D, 0.7))
    scale = max(1.0, np.abs(go).max())
    assert np.abs(out[0] - go).max() <= 1e-10 * scale
    assert np.abs(out[0] - out[1]).max() <= 1e-10 * scale
    assert np.abs(out[0].sum(0)).max() <= 1e-10 * scale
