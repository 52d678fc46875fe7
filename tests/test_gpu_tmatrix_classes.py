"""The solve by parity classes at the edges of its shared-memory groups: for a lossless spheroid
the T-matrix of a mode is that of a lossless scatterer, T + T^H + 2 T^H T = 0 (S = 1 + 2 T
unitary), and elements of opposite parity of (element + order) are exactly zero. Tolerance: the
truncated T at n_theta = 2 N holds its unitarity to the quadrature's and the refinement's floor;
1e-9 is the converged records' (test_gpu_tmatrix)."""

import numpy as np
import pytest

from scatrs_b200 import _native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("unknowns", [1, 2, 3, 35, 36, 37, 56, 57, 80, 81, 112, 113])
def test_unitarity_across_groups(gpu, unknowns):
    mode = 3
    n = unknowns + mode - 1
    t = _native.spheroid_tmatrix(18.0 if unknowns > 30 else 0.3, 1.2, 1.4 + 0.0j, mode, n,
                                 max(2 * n, 24))
    k = unknowns
    assert t.shape == (2 * k, 2 * k) and np.all(np.isfinite(t.view(np.float64)))
    f = np.arange(2 * k)
    parity = (f % k + f // k) % 2
    assert np.all(t[parity[:, None] != parity[None, :]] == 0.0)
    r = t + t.conj().T + 2.0 * t.conj().T @ t
    assert np.abs(r).max() <= 1e-9
