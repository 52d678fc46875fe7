"""Chunks on the phase levels (their elements at 2 U + 1 Gauss nodes, interpolated onto the
requested cosines) against the oracle's direct sums, at the levels' edges and for the cosine lists
a caller may pass. Tolerance: as the direct path's and in its measure (test_gpu_ensemble: 1e-12 of
max F11 and of the largest alpha_1; the oracle's own alpha are 8e-12 from extended precision at 255
terms, 9e-14 of the largest): the elements are
polynomials of degree at most 2 U, so the interpolation is exact up to rounding, and the Lagrange
functions of Gauss nodes sum to at most about 13 in magnitude."""

import numpy as np
import pytest

from oracle import oracle as O
from scatrs_b200 import _native
from scatrs_b200 import workloads as W

pytestmark = pytest.mark.gpu

TOL = 1e-12


def _x_of_terms(n):
    """A size parameter whose truncation ceil(x + 6 x^(1/3) + 3) is n."""
    lo, hi = 1e-3, float(n)
    for _ in range(200):
        mid = 0.5 * (lo + hi)
        lo, hi = (mid, hi) if np.ceil(mid + 6 * np.cbrt(mid) + 3) < n else (lo, mid)
    return hi * (1 + 1e-9)


def _check(dists, wl, m, n_nodes, mu, order, i8_above=0, tol=TOL):
    v, ph, g = _native.ensemble_fixed(dists, wl, m, mu, n_nodes, order, i8_above=i8_above)
    d = np.zeros(dists.size, dtype=O.DIST_DTYPE)
    d["kind"], d["p"] = dists["kind"], dists["param"]
    d["r_lo"], d["r_hi"] = dists["r_lo"], dists["r_hi"]
    ref = O.ensemble_fixed(d, wl, m, n_nodes, mu, order if order >= 0 else None)
    np.testing.assert_allclose(v[:2], ref["values"][:2], rtol=tol)
    size = np.abs(ref["phase"][0]).max(axis=1, keepdims=True)
    assert np.max(np.abs(ph - ref["phase"]) / size[None]) <= tol
    if order >= 0:
        scale = np.abs(ref["greek"][0]).max(axis=1, keepdims=True)
        assert np.max(np.abs(g - ref["greek"]) / scale[None]) <= tol


@pytest.mark.parametrize("terms", [8, 31, 32, 63, 64, 255, 256, 300])
@pytest.mark.parametrize("order", [-1, 7, 64])
def test_level_edges(gpu, terms, order):
    wl = np.array([0.5])
    r = _x_of_terms(terms) * wl[0] / (2 * np.pi)
    d = W.lognormals([0.8 * r], [1.3], 1)
    d["r_lo"], d["r_hi"] = 0.6 * r, r * (1 + 1e-6)
    m = np.array([[1.45 + 0.01j]])
    _check(d, wl, m, 45, _native.gauss_legendre(200)[0], order)


@pytest.mark.parametrize("mu", [
    np.array([-1.0, -0.0, 0.3, 1.0]),
    np.array([0.5]),
    np.linspace(-1.0, 1.0, 181),
    np.concatenate([np.cos(np.radians(np.arange(0.0, 90.0, 0.5))), [0.25, 0.25, -0.25]]),
    _native.gauss_legendre(63)[0],  # the first level's own nodes
], ids=["ends", "one", "degrees", "unpaired", "nodes"])
def test_cosine_lists(gpu, mu):
    d = W.lognormals([0.05, 0.4], [1.5, 1.8], 3)
    wl = np.array([0.4, 1.1])
    m = np.array([[1.5 + 1e-3j, 1.4 + 1e-6j], [1.33 + 0.1j, 1.6 + 0.0j]])
    _check(d, wl, m, 150, mu, 20)


def test_levels_grow_and_share(gpu):
    # Small then large inputs on the same context, and the other way round.
    mu = _native.gauss_legendre(90)[0]
    wl = np.array([0.55])
    m = np.array([[1.4 + 1e-4j]])
    for median in (0.02, 2.0, 0.1, 4.0, 0.02):
        _check(W.lognormals([median], [1.4], 3), wl, m, 96, mu, 16)


def test_mixed_form_on_levels(gpu):
    d = W.lognormals([0.6], [1.6], 3)
    wl = np.array([0.4, 0.9])
    _check(d, wl, np.full((1, 2), 1.5 + 1e-3j), 256, _native.gauss_legendre(180)[0], 32,
           i8_above=16, tol=1e-10)
