"""The FP64 pair functions over the range of their table (from r = a/2 on) against 50
digits: isolated pairs at exact distances, forces along and across the line of centres.
Tolerance 1e-14 of |F| + |G|: the closed form in FP64 has terms up to 8 times that, each
of a few roundings (90 of 2^-53)."""
from decimal import Decimal as D, getcontext

import numpy as np
import pytest

import spme_gb300

pytestmark = pytest.mark.gpu


def _erf(x):
    """sum of (-1)^k x^(2k+1) / (k! (2k+1)), times 2/sqrt(pi) by the caller."""
    s, t, k = D(0), x, 0
    while abs(t) > D(10) ** -70:
        s += t / (2 * k + 1)
        k += 1
        t *= -x * x / k
    return s


def _pair(r, xi, a):
    """F and G of M_real = F I + G r r^T / r^2."""
    getcontext().prec = 50
    r, xi, a = D(r), D(xi), D(a)
    pi = D("3.14159265358979323846264338327950288419716939937510582")
    rsp = 1 / pi.sqrt()
    x = xi * r
    x2 = x * x
    e = (-x2).exp() * rsp
    ef = 2 * rsp * _erf(x)
    c1, c3, ic = D("0.75"), D("0.5"), 1 - ef
    f = ic * (c1 / r + c3 * a * a / r ** 3) + e * (
        4 * xi ** 7 * a * a * r ** 4 + 3 * xi ** 3 * r * r - 20 * xi ** 5 * a * a * r * r
        - D("4.5") * xi + 14 * xi ** 3 * a * a + xi * a * a / (r * r))
    g = ic * (c1 / r - 3 * c3 * a * a / r ** 3) + e * (
        -4 * xi ** 7 * a * a * r ** 4 - 3 * xi ** 3 * r * r + 16 * xi ** 5 * a * a * r * r
        + D("1.5") * xi - 2 * xi ** 3 * a * a - 3 * xi * a * a / (r * r))
    if r < 2 * a:  # overlap form minus the far form
        f += (1 - 9 * r / (32 * a)) / a - c1 / r - c3 * a * a / r ** 3
        g += 3 * r / (32 * a * a) - c1 / r + 3 * c3 * a * a / r ** 3
    return f, g


@pytest.mark.parametrize("xi", [0.2, 0.3, 0.5])
def test_against_50_digits(gpu_lib, xi):
    # 16 cells of edge 32 per axis (the cap for 520 particles), a pair in every other one
    L, rc, a, n = 512.0, 20.0, 1.0, 520
    m = n // 2
    r = np.round(np.exp(np.linspace(np.log(0.5 * a + 1e-3), np.log(min(rc - 1e-3, 4 / xi)), m))
                 * 2 ** 20) / 2 ** 20
    site = 64.0 * np.stack(np.unravel_index(np.arange(m), (8, 8, 8)), 1) + [2.0, 3.0, 5.0]
    pos = np.concatenate([site, site])
    pos[m:, 0] += r
    f = np.zeros((2, n, 3))
    f[0, m:, 0] = f[1, m:, 1] = 1.0
    eng = spme_gb300.Engine(n, L, xi, 16, 4, radius=a, rcut=rc, precision="fp64", max_nrhs=2,
                            terms=spme_gb300.TERM_REAL)
    eng.set_positions(pos)
    u = eng.apply(f.reshape(2, 3 * n)).reshape(2, n, 3)
    eng.close()
    for i in range(m):
        F, G = _pair(float(r[i]), xi, a)
        tol = D("1e-14") * (abs(F) + abs(G))
        assert abs(D(float(u[1, i, 1])) - F) < tol, r[i]
        assert abs(D(float(u[0, i, 0])) - F - G) < tol, r[i]
