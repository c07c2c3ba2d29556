"""The device Rys rule at the edges of its tables' intervals (half-unit steps
for one and two roots, unit steps above) and at the switch to the large-T
limit, against 60-digit rules from the Boys moments.

Tolerance: the tables are within 3e-16 of the exact rule (binary128 fits,
reported by their generator), evaluation in double adds a few ulp, and the
large-T limit starts where it agrees with the exact rule to 2e-15: 4e-15."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
mp = pytest.importorskip("mpmath")

TASYM = {1: 36, 2: 44, 3: 50, 5: 63, 7: 74}


def rule_mp(n, T):
    mp.mp.dps = 60
    T = mp.mpf(float(T))

    def boys(k):
        a = k + mp.mpf(1) / 2
        return 1 / (2 * a) if T == 0 else mp.gammainc(a, 0, T) / (2 * T ** a)
    m = [boys(k) for k in range(2 * n + 1)]
    H = mp.matrix(n + 1, n + 1)
    for i in range(n + 1):
        for j in range(n + 1):
            H[i, j] = m[i + j]
    R = mp.cholesky(H).T
    J = mp.matrix(n, n)
    for i in range(n):
        J[i, i] = R[i, i + 1] / R[i, i] - (R[i - 1, i] / R[i - 1, i - 1] if i else 0)
        if i + 1 < n:
            J[i, i + 1] = J[i + 1, i] = R[i + 1, i + 1] / R[i, i]
    E, Q = mp.eighe(J)
    order = sorted(range(n), key=lambda i: E[i])
    return [E[i] for i in order], [m[0] * Q[0, i] ** 2 for i in order]


@pytest.mark.parametrize("n", [1, 2, 3, 5, 7])
def test_interval_edges(n):
    import iqcp_b200 as iq
    ta = float(TASYM[n])
    edges = [0.5, 1.0, 1.5, 7.0, 20.5, ta - 0.5, ta]
    T = np.array([0.0, 1e-9, 0.25] + [t for e in edges for t in (np.nextafter(e, 0), e, np.nextafter(e, 100))] + [ta + 9.3])
    R, W = iq.rys_roots(n, T)
    for i, t in enumerate(T):
        x, w = rule_mp(n, t)
        for k in range(n):
            assert abs(float((mp.mpf(float(R[i, k])) - x[k]) / x[k])) < 4e-15, (t, k)
            assert abs(float((mp.mpf(float(W[i, k])) - w[k]) / w[k])) < 4e-15, (t, k)
