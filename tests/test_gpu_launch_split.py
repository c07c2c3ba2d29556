"""J/K and gradient launches that fill the chip many times over set their own
split of an SM's memory, short ones leave it to the driver: 40 atoms (long
launches of the small classes) and benzene (short ones), called directly and
replayed from a captured graph.

Tolerance: the same sums in another order of atomic additions, 1e5 of them at
1e-16 each, 1e-11 relative to the largest element."""
import numpy as np
import pytest
import torch

from conftest import random_density
from iqcp_b200 import BasisSet, FockEngine
from iqcp_b200.molecules import REFERENCE_MOLECULES, workload

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("large", [False, True])
def test_captured_launches(large):
    atoms, basis = workload("c2", 0) if large else (REFERENCE_MOLECULES["C6H6"], "6-31g*")
    b = BasisSet.build(atoms, basis)
    n = b.n_basis
    D = torch.from_numpy(random_density(n, 3, 0.2)).cuda()
    st = torch.cuda.Stream()
    out = [torch.empty(2, n, n, dtype=torch.float64, device="cuda") for _ in range(2)]
    grad = [torch.zeros(b.n_atoms, 3, dtype=torch.float64, device="cuda") for _ in range(2)]
    with FockEngine(b) as eng:
        eng.set_stream(st.cuda_stream)

        def call(i):
            eng.jk_device(D.data_ptr(), out[i][0].data_ptr(), out[i][1].data_ptr())
            eng.eri_gradient_device(D.data_ptr(), 1.0, grad[i].data_ptr())

        st.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(st):
            call(0)
            st.synchronize()
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g, stream=st):
                call(1)
            g.replay()
            st.synchronize()
        del g
    for x, y in (*zip(out[0], out[1]), (grad[0], grad[1])):
        x, y = x.cpu().numpy(), y.cpu().numpy()
        assert np.abs(x).max() > 0
        assert np.abs(x - y).max() <= 1e-11 * np.abs(x).max()
