"""Q_sca of lossless spheroids against their T-matrices' own sums: an excess over Q_ext beyond
rounding (a truncation too small) is reported, one within rounding is not."""

import numpy as np
import pytest

from scatrs_b200 import _native

pytestmark = pytest.mark.gpu

# Sums of up to 4 N^2 squares per mode, in another order than the kernel's: a few hundred ulps.
TOL = 1e-13


def _sums(x, eps, m, n, n_theta):
    ext = sca = 0.0
    for mode in range(n + 1):
        t = _native.spheroid_tmatrix(x, eps, m, mode, n, n_theta)
        w = 1.0 if mode == 0 else 2.0
        ext -= w * np.trace(t).real
        sca += w * np.sum(np.abs(t) ** 2)
    return 2.0 / x ** 2 * ext, 2.0 / x ** 2 * sca


def test_an_energy_excess_is_reported(gpu):
    excess = []
    for x, eps, n, n_theta in [(4.0, 2.0, 6, 8), (4.0, 0.5, 6, 8), (6.0, 2.5, 8, 10),
                               (6.0, 0.4, 8, 10), (3.0, 3.0, 5, 6), (5.0, 1.5, 7, 8),
                               (5.0, 1.7, 6, 7), (2.0, 2.5, 4, 5)]:
        r = gpu.spheroid_compute(np.array([x]), eps, 1.5 + 0j, n_terms=n, n_theta=n_theta)
        q_ext, q_sca, q_abs = r["efficiencies"][0][:3]
        ext, sca = _sums(x, eps, 1.5 + 0j, n, n_theta)
        assert abs(q_ext - ext) <= TOL * ext and abs(q_sca - sca) <= TOL * ext
        assert q_abs == q_ext - q_sca
        excess.append((sca - ext) / ext)
    assert max(excess) > 1e-9, excess  # some of them scatter more than they extinguish


def test_rounding_alone_is_not(gpu):
    x = np.linspace(0.5, 6.0, 24)
    q = gpu.spheroid_compute(x, 1.5, 1.5 + 0j, rtol=1e-8)["efficiencies"]
    assert (q[:, 1] <= q[:, 0]).all() and (q[:, 0] - q[:, 1] <= 64 * 2.0 ** -52 * q[:, 0]).all()
