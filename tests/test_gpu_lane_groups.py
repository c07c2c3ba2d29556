"""Quartets shared by groups of lanes: contractions from one primitive per
shell to nine (1 to 6561 primitive quartets per quartet, groups of 1 to 32
lanes), a ket bucket's remainder spread over idle lanes, single contexts and
batches, every gradient variant that runs in lane groups, and the mixed form's
FP32 share.

Tolerances: both sides transfer angular momentum to the second centre
horizontally, which for exponents up to 60 on centres 2 bohr apart costs
2e-16 * AB^2 * 2p ~ 1e-13 per transfer, squared over bra and ket d shells; 1e-10
relative to the largest element holds that with an order to spare (the oracle's
roots in extended precision).  FP32 quadrature: 6e-8 times the same transfer
loss per index, 1e-3."""
import numpy as np
import pytest

from conftest import random_density
from iqcp_b200 import MIXED, BasisSet, BatchFockEngine, FockEngine

pytestmark = pytest.mark.gpu


def deep(n, centres, ls):
    """Shells of n primitives of the given angular momenta on a few centres."""
    rng = np.random.default_rng(n)
    xyz = np.array([[0, 0, 0.1], [1.3, -0.4, 0.2], [-0.7, 1.1, 0.9], [0.4, -1.2, -0.8]])[:centres]
    at = np.repeat(np.arange(centres), len(ls))
    ex = np.geomspace(0.3, 60.0, n) if n > 1 else np.array([0.7])
    return BasisSet("deep", [2] * centres, xyz, list(ls) * centres, [n] * len(at), at, xyz[at],
                    ex.tolist() * len(at), rng.uniform(0.1, 0.4, n * len(at)))


@pytest.fixture(scope="module")
def refs(oracle_mod):
    out = {}
    oracle_mod.set_root_precision(True)
    try:
        for n, c, ls in ((1, 3, (0, 1, 2)), (3, 2, (0, 1, 2)), (6, 2, (0, 1)), (9, 2, (0, 1))):
            b = deep(n, c, ls)
            D = random_density(b.n_basis, n)
            J, K, _ = oracle_mod.jk_direct(b, D)
            g, _ = oracle_mod.eri_gradient(b, D, 1.0)
            out[n] = (b, D, J, K, g)
    finally:
        oracle_mod.set_root_precision(False)
    return out


def close(a, ref, tol=1e-10):
    assert np.abs(np.asarray(a) - ref).max() <= tol * max(1.0, np.abs(ref).max())


@pytest.mark.parametrize("mode", [0, 2, 3])
@pytest.mark.parametrize("n", [1, 3, 6, 9])
def test_against_oracle(refs, n, mode):
    b, D, Jo, Ko, go = refs[n]
    with FockEngine(b) as eng:
        eng.set_kernel_mode("jk", mode=0)
        eng.set_kernel_mode("grad", mode=mode)
        J, K = eng.build_jk(D)
        g = eng.eri_gradient(D, 1.0)
    close(J, Jo)
    close(K, Ko)
    close(g, go)


def test_batch_of_unequal_contractions(refs):
    use = [refs[n] for n in (6, 1, 3, 6)]
    with BatchFockEngine([r[0] for r in use]) as eng:
        eng.set_kernel_mode("jk", mode=0)
        eng.set_kernel_mode("grad", mode=0)
        J, K = eng.build_jk([r[1] for r in use])
        g = eng.eri_gradient([r[1] for r in use])
    for m, r in enumerate(use):
        close(J[m], r[2])
        close(K[m], r[3])
        close(g[m], r[4])


@pytest.mark.parametrize("n", [3, 6])
def test_fp32_share(refs, n):
    b, D, Jo, Ko, go = refs[n]
    with FockEngine(b, precision=MIXED, mixed_cutoff=1e30) as eng:
        for kind in ("jk32", "grad32"):
            eng.set_kernel_mode(kind, mode=0)
        J, K = eng.build_jk(D)
        g = eng.eri_gradient(D, 1.0)
    close(J, Jo, 1e-3)
    close(K, Ko, 1e-3)
    close(g, go, 1e-3)
