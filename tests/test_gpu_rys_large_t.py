"""The large-T limit of the device's Rys rule: the roots are c / T and the weights
c / sqrt(T) with the tabulated constants c.

Tolerances: one rounding (2^-53) for a root, which is a division; the reciprocal
square root is within one unit in the last place (2^-52) and its product rounds
once more, 3 2^-53 for a weight."""
import os
import re

import numpy as np
import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu
mp = pytest.importorskip("mpmath")
TASYM = {1: 36, 2: 44, 3: 50, 4: 57, 5: 63, 6: 68, 7: 74}


def _table(name):
    with open(os.path.join(ROOT, "iqcp_b200", "csrc", "rys_tables.inc")) as f:
        body = re.search(name + r"\[[^\]]*\] = \{([^}]*)\}", f.read()).group(1)
    return [float(x) for x in body.replace("\n", " ").split(",") if x.strip()]


@pytest.mark.parametrize("n", sorted(TASYM))
def test_roots_and_weights_of_the_limit(n):
    import iqcp_b200 as iq
    mp.mp.dps = 40
    c, w = _table("kRysAsymRoot"), _table("kRysAsymWeight")
    base = n * (n - 1) // 2
    rng = np.random.default_rng(n)
    T = np.concatenate([[TASYM[n], np.nextafter(TASYM[n], 1e9)], np.exp(rng.uniform(np.log(TASYM[n]), np.log(1e9), 500))])
    R, W = iq.rys_roots(n, T)
    for i, t in enumerate(T):
        t = mp.mpf(float(t))
        for k in range(n):
            r, v = mp.mpf(c[base + k]) / t, mp.mpf(w[base + k]) / mp.sqrt(t)
            assert abs(mp.mpf(float(R[i, k])) - r) <= 1.001 * 2.0 ** -53 * r, (n, float(t), k)
            assert abs(mp.mpf(float(W[i, k])) - v) <= 3.001 * 2.0 ** -53 * v, (n, float(t), k)


def test_largest_arguments_stay_finite():
    import iqcp_b200 as iq
    for n in sorted(TASYM):
        R, W = iq.rys_roots(n, np.array([1e200, np.finfo(float).max]))
        assert np.isfinite(R).all() and np.isfinite(W).all() and (R >= 0).all() and R.max() < 1e-197 and W.max() < 1e-99
