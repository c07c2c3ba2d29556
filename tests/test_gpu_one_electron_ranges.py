"""One-electron kernels at the sizes where their work distribution changes:
more primitive pairs than a warp stages at once, molecules of one atom up to
more atoms than lanes, and a batch of more atoms than one launch takes.

Tolerance: sums of a few thousand FP64 terms of mixed sign, each exact to a few
ulp; 1e-11 relative to the largest element leaves two orders for cancellation."""
import numpy as np
import pytest

from conftest import random_density
from iqcp_b200 import BasisSet, BatchFockEngine, FockEngine
from iqcp_b200.molecules import REFERENCE_MOLECULES, workload

pytestmark = pytest.mark.gpu


def check(oracle_mod, b, seed):
    D, W = random_density(b.n_basis, seed), random_density(b.n_basis, seed + 1)
    with FockEngine(b) as eng:
        mats = eng.one_electron()
        g = eng.one_electron_gradient(D, W)
    for name, M in zip("STV", mats):
        Mo = oracle_mod.one_electron(b, name)
        assert np.abs(M - Mo).max() <= 1e-11 * max(1.0, np.abs(Mo).max()), name
    go = oracle_mod.one_electron_gradient(b, D, W)
    assert np.abs(g - go).max() <= 1e-11 * max(1.0, np.abs(go).max())


def deep(n):
    """s, p and d shells of n primitives on three centres (n * n primitive pairs)."""
    rng = np.random.default_rng(n)
    xyz = np.array([[0, 0, 0.1], [1.3, -0.4, 0.2], [-0.7, 1.1, 0.9]])
    l = [0, 1, 2] * 3
    at = np.repeat(np.arange(3), 3)
    return BasisSet("deep", [8, 6, 1], xyz, l, [n] * 9, at, xyz[at], np.geomspace(0.2, 900.0, n).tolist() * 9,
                    rng.uniform(0.05, 0.4, 9 * n))


@pytest.mark.parametrize("n", [1, 5, 6, 9])
def test_primitive_pairs_per_stage(oracle_mod, n):
    check(oracle_mod, deep(n), 3 + n)


@pytest.mark.parametrize("mol", ["He", "H2", "CH4", "c2"])
def test_atoms_per_warp(oracle_mod, mol):
    if mol == "c2":
        atoms, basis = workload("c2")[0], "sto-3g"
    else:
        atoms, basis = REFERENCE_MOLECULES.get(mol, [(2, (0.1, 0.2, -0.3))]), "6-31g*"
    check(oracle_mod, BasisSet.build(atoms, basis), 11)


def test_more_atoms_than_a_launch():
    """700 water molecules (2100 atoms): two launches, same results as one context each."""
    h2o = REFERENCE_MOLECULES["H2O"]
    bases = [BasisSet.build([(z, tuple(np.array(x) + 0.01 * m)) for z, x in h2o], "sto-3g") for m in range(700)]
    D = random_density(bases[0].n_basis, 5)
    with BatchFockEngine(bases) as eng:
        S, T, V = eng.one_electron()
        g = eng.one_electron_gradient([D] * 700, [0.5 * D] * 700)
    for m in (0, 681, 682, 683, 699):
        with FockEngine(bases[m]) as one:
            for M, Mo in zip((S[m], T[m], V[m]), one.one_electron()):
                assert np.abs(M - Mo).max() < 1e-12
            assert np.abs(g[m] - one.one_electron_gradient(D, 0.5 * D)).max() < 1e-11
