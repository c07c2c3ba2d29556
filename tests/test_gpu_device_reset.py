"""Contexts made after the process has reset the device, in a process of their own:
what the library keeps between contexts belongs to the old CUDA context."""
import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

SCRIPT = """
import ctypes
import numpy as np
import torch
from iqcp_b200 import BasisSet, FockEngine
from iqcp_b200.batch_scf import BatchRHF
from iqcp_b200.molecules import REFERENCE_MOLECULES

maps = open("/proc/self/maps").read().split()
cudart = ctypes.CDLL(next(p for p in maps if "libcudart" in p))
bases = [BasisSet.build(REFERENCE_MOLECULES[m], "6-31g*") for m in ("H2O", "C6H6")]


def figures():
    out = []
    for b in bases:
        D = np.eye(b.n_basis) + 0.1
        with FockEngine(b) as eng:      # C6H6: kernels above the default shared-memory limit
            out += list(eng.build_jk(D)) + [eng.eri_gradient(D)]
            p = []
            for n in (1, 1, 1):
                p.append(ctypes.c_void_p())
                assert cudart.cudaMalloc(ctypes.byref(p[-1]), D.nbytes) == 0
            cudart.cudaMemcpy(p[0], D.ctypes.data_as(ctypes.c_void_p), D.nbytes, 1)
            eng.jk_device_noalloc(p[0].value, p[1].value, p[2].value)
            cudart.cudaDeviceSynchronize()
            for q in p[1:]:
                x = np.empty_like(D)
                cudart.cudaMemcpy(x.ctypes.data_as(ctypes.c_void_p), q, D.nbytes, 2)
                out.append(x)
            for q in p:
                cudart.cudaFree(q)
    scf = BatchRHF(bases[:1])
    out.append(scf.run(e_tol=1e-11, d_tol=1e-9, err_tol=1e-8).energies)
    scf.close()
    return out


ref = figures()
for _ in range(2):
    stale = FockEngine(bases[0])
    assert cudart.cudaDeviceReset() == 0
    if _ == 0:
        stale.close()
    got = figures()
    assert max(np.abs(x - y).max() for x, y in zip(ref, got)) < 1e-10
    stale.close()
print("same figures")
"""


def test_contexts_after_a_device_reset():
    r = subprocess.run([sys.executable, "-c", SCRIPT], cwd=ROOT, env=dict(os.environ, PYTHONPATH=ROOT),
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "same figures" in r.stdout, r.stdout + r.stderr
