"""K-a with a block per chunk (few chunks, mie_split_kernel) against a warp per chunk (the same units
among many others): the same bits, at chunks of fewer orders than warps, of lossless particles and
at the ends of the warps' runs."""

import numpy as np
import pytest

from scatrs_b200 import _native
from scatrs_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("median", [1e-4, 0.02, 0.3, 4.0])
@pytest.mark.parametrize("k", [0.0, 1e-3])
def test_same_bits_as_a_warp_per_chunk(gpu, median, k):
    n_fill = 3000  # units of 4 chunks: more than a slab splits
    d = W.lognormals([median], [1.5], 2)
    wl = np.array([0.6])
    m = np.array([[1.45 + 1j * k]])
    mu = np.array([-0.7, 0.1, 0.9])
    few = _native.ensemble_fixed(d, wl, m, mu, 100, 8)
    filled = np.concatenate([d, W.lognormals(np.full(n_fill, median), 1.5, 2)])
    many = _native.ensemble_fixed(filled, wl, np.full((n_fill + 1, 1), m[0, 0]), mu, 100, 8)
    for a, b in zip(few, many):
        assert np.array_equal(a[:, 0], b[:, 0])
