"""Phase levels in the backward directions, relative to their own values: F11 of one sphere there is
orders of magnitude below the forward peak, and interpolation must be no further off than sums on
tables at the requested cosines themselves (the oracle's form, double recurrences)."""

import math

import numpy as np
import pytest

from scatrs_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _tables(mu, n_max, real):
    """(2n + 1) / (n (n + 1)) times pi_n and tau_n, n = 1..n_max, in the given precision."""
    mu = mu.astype(real)
    prev, cur = np.zeros_like(mu), np.ones_like(mu)
    p, t = [], []
    for n in range(1, n_max + 1):
        n0, n1 = real(n), real(n + 1)
        w = real(2 * n + 1) / (n0 * n1)
        p.append(w * cur)
        t.append(w * (n0 * mu * cur - n1 * prev))
        prev, cur = cur, (real(2 * n + 1) * mu * cur - n1 * prev) / n0
    return np.array(p).T, np.array(t).T


def _f11(mu, a, b, real, cplx):
    p, t = _tables(mu, a.size, real)
    s1 = p.astype(cplx) @ a.astype(cplx) + t.astype(cplx) @ b.astype(cplx)
    s2 = t.astype(cplx) @ a.astype(cplx) + p.astype(cplx) @ b.astype(cplx)
    return (s1.real ** 2 + s1.imag ** 2 + s2.real ** 2 + s2.imag ** 2) / 2


@pytest.mark.parametrize("x,n_mu", [(30.0, 360), (100.0, 360), (300.0, 1200)])
def test_backward_values(gpu, x, n_mu):
    wl, m = np.array([0.5]), np.array([[1.33 + 1e-4j]])
    d = W.lognormals([x * wl[0] / (2 * np.pi)], [1.2], 1)
    # The grid's single node, and the coefficients there, as the library forms them.
    r = math.exp(0.5 * (math.log(d["r_lo"][0]) + math.log(d["r_hi"][0])))
    xs = 2.0 * math.pi * r / wl[0]
    (a, b), = gpu.mie(np.array([xs]), m[0])[0]
    mu = np.cos((np.arange(n_mu) + 0.5) * np.pi / n_mu)
    _, ph, _ = gpu.ensemble_fixed(d, wl, m, mu, 1, normalized=False)
    got = ph[0, 0] / (4.0 / (xs * xs) * (math.pi * r * r))
    back = mu < -0.02
    want = _f11(mu[back], a, b, np.longdouble, np.clongdouble)
    direct = _f11(mu[back], a, b, np.float64, np.complex128)
    off = np.abs(got[back] - want) / want
    assert off.max() <= (np.abs(direct - want) / want).max(), off.max()
