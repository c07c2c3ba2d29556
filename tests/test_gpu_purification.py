"""Density purification of the batched SCF on both sides of its size rule (one
kernel per step up to 160 functions, batched products above), at block edges and
for the smallest matrices: the same energies, densities and gradients whichever
molecules share the batch.

Tolerances: both forms stop at idempotency to 1e-13 in the trace, and the SCF is
converged to dE 1e-10, rms dD 1e-9: 1e-9 in energy, 1e-7 in density elements."""
import numpy as np
import pytest

from iqcp_b200 import BasisSet
from iqcp_b200.batch_scf import BatchRHF
from iqcp_b200.molecules import REFERENCE_MOLECULES, generate

pytestmark = pytest.mark.gpu

SMALL = [("H2", "sto-3g"), ("HF", "6-31g"), ("CH4", "6-31g*"), ("H2O", "cc-pvdz"), ("C6H6", "6-31g*"), ("C6H6", "cc-pvdz")]


def run(bases):
    rhf = BatchRHF(bases)
    r = rhf.run(e_tol=1e-10, d_tol=1e-9, err_tol=1e-7, D0=rhf.sad_guess())
    out = (r.energies, rhf.densities(), rhf.gradients(), r.converged)
    rhf.close()
    return out


def test_small_step_and_batched_products_agree():
    bases = [BasisSet.build(REFERENCE_MOLECULES[m], b) for m, b in SMALL]
    assert sorted(b.n_basis for b in bases)[0] == 2 and max(b.n_basis for b in bases) <= 160
    big = BasisSet.build(generate(22, (6, 7, 8), 12, 0), "6-31g*")
    assert big.n_basis > 160
    E, D, g, conv = run(bases)
    Eb, Db, gb, convb = run(bases + [big])
    assert conv.all() and convb[: len(bases)].all()
    for k in range(len(bases)):
        assert abs(E[k] - Eb[k]) < 1e-9
        assert np.abs(D[k] - Db[k]).max() < 1e-7
        assert np.abs(g[k] - gb[k]).max() < 1e-6


@pytest.mark.parametrize("mol,basis", SMALL)
def test_density_is_a_projector(mol, basis):
    """D S D = 2 D, Tr D S = electrons."""
    b = BasisSet.build(REFERENCE_MOLECULES[mol], basis)
    rhf = BatchRHF([b])
    r = rhf.run(D0=rhf.sad_guess())
    D = rhf.densities()[0]
    S = rhf.eng.one_electron()[0][0]
    rhf.close()
    assert r.converged.all()
    assert abs(np.sum(D * S) - b.n_electrons) < 1e-9
    assert np.abs(D @ S @ D - 2 * D).max() < 1e-9 * max(1.0, np.abs(D).max())
