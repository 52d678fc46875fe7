"""Calls at the ends of what the entry points take."""

import numpy as np
import pytest

from scatrs_b200 import workloads as W

pytestmark = pytest.mark.gpu

WL, M = np.array([0.5]), np.array([[1.45 + 1e-3j]])


def _droplet():
    return W.lognormals([0.2], [1.3], 2)


@pytest.mark.parametrize("order", [1 << 20, 1 << 21])
def test_greek_orders_to_the_limit(gpu, order):
    _, ph0, g0 = gpu.ensemble_fixed(_droplet(), WL, M, W.gauss_legendre(60), 32, 200)
    _, ph, g = gpu.ensemble_fixed(_droplet(), WL, M, W.gauss_legendre(60), 32, order)
    # The coefficients end at twice the largest number of terms: the same tables, the same bits.
    assert np.array_equal(ph, ph0) and np.array_equal(g[..., :201], g0)
    assert not g[..., 201:].any() and g0[0, 0, 1:8].all() and not g0[..., 150:].any()


def test_cosines_beyond_the_grids_rows(gpu):
    # 2^21 rows are 65,536 tiles of one phase level's interpolation.
    n = 1 << 21
    mu = np.cos(np.linspace(0.0, np.pi, n) * (1 - 1e-9))
    at = np.r_[0:8, n // 2:n // 2 + 8, n - 40:n]
    d = W.lognormals([0.05], [1.2], 2)
    _, ph, _ = gpu.ensemble_fixed(d, WL, M, mu, 32)
    _, want, _ = gpu.ensemble_fixed(d, WL, M, mu[at], 32)
    assert np.max(np.abs(ph[..., at] - want)) <= 1e-12 * want[0].max()


def test_more_spheroids_than_grid_rows(gpu):
    # 70,000 spheroids of one truncation in a call: every one as on its own.
    n = 70_000
    x = np.full(n, 0.3)
    x[::7], x[-1] = 0.2, 0.25
    got = gpu.spheroid_compute(x, 1.5, 1.5 + 1e-2j, n_terms=2, n_theta=4, greek_order=2)
    for v in (0.2, 0.25, 0.3):
        want = gpu.spheroid_compute(np.array([v]), 1.5, 1.5 + 1e-2j, n_terms=2, n_theta=4,
                                    greek_order=2)
        assert (got["efficiencies"][x == v] == want["efficiencies"][0]).all()
        assert (got["greek"][x == v] == want["greek"][0]).all()


def test_no_errors_before_the_first_ensemble_call(gpu):
    lib = gpu.load()
    lib.scatrs_release()
    gpu.check_errors()
    lib.scatrs_release()
    gpu.mie(np.array([1.0]), np.array([1.5 + 0j]))
    gpu.check_errors()
