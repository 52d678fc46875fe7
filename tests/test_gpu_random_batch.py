"""The orientation average with its shared coefficient tables: spheroids of different truncations
in one call, in either order (the tables grow on the way), against calls of their own. The
per-spheroid sums do not depend on the batch, so the results agree bit for bit."""

import numpy as np
import pytest

from scatrs_b200 import _native

pytestmark = pytest.mark.gpu

X = np.array([0.2, 1.0, 2.5, 4.0, 7.5, 11.0])
EPS = np.array([1.5, 0.7, 2.0, 1.0, 0.8, 1.3])
M = np.array([1.5 + 0.01j, 1.33 + 0j, 1.6 + 0.1j, 1.45 + 1e-3j, 1.5 + 0.02j, 1.4 + 1e-4j])


@pytest.mark.parametrize("order", ["ascending", "descending"])
def test_batches_equal_single_calls(gpu, order):
    at = np.arange(X.size) if order == "ascending" else np.arange(X.size)[::-1]
    batch = _native.spheroid_compute(X[at], EPS[at], M[at], rtol=1e-8, greek_order=12)
    for k, i in enumerate(at):
        one = _native.spheroid_compute(X[i], EPS[i], M[i], rtol=1e-8, greek_order=12)
        assert np.array_equal(batch["greek"][k], one["greek"][0])
        assert np.array_equal(batch["efficiencies"][k], one["efficiencies"][0])
