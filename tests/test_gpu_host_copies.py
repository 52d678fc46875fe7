"""The copies between the host and the device that go block by block through pinned staging: the
outputs of a host call at lengths about the copy's threshold (256 KiB) and its blocks (2 MiB), and
the adaptive node tables of more records than a block of 8 MiB holds."""

import numpy as np
import pytest

from oracle import oracle as O
from scatrs_b200 import _native
from scatrs_b200 import workloads as W
from test_gpu_adaptive import MU, _compare, _dists, _odist

pytestmark = pytest.mark.gpu


# 3 cosines: 144 B of phase matrix a unit.
@pytest.mark.parametrize("n", [1, 1820, 1821, 14563, 14564, 30011])
def test_outputs_land_at_their_units(gpu, n):
    period = 7  # no divisor of a block: a block at the wrong place shows
    median = 0.05 * (1 + np.arange(n) % period)
    d = W.lognormals(median, 1.4, 2)
    wl = np.array([0.6])
    m = np.full((n, 1), 1.4 + 0.01j)
    out = _native.ensemble_fixed(d, wl, m, np.array([-0.5, 0.2, 1.0]), 8, 4)
    one = _native.ensemble_fixed(d[:period], wl, m[:period], np.array([-0.5, 0.2, 1.0]), 8, 4)
    for a, b in zip(out, one):
        assert np.array_equal(a, b[:, np.arange(n) % period])


def test_node_records_of_several_blocks(gpu):
    n = 500
    rng = np.random.default_rng(7)
    specs = [(5, 0.3) if k % 97 == 5 else (1, float(rng.uniform(0.05, 0.8)), 1.6)
             for k in range(n)]
    wl = np.array([0.35, 0.55, 1.0, 2.0])
    m = np.array([1.43 + 1e-8j, 1.5 + 0.01j, 1.33 + 0.0j, 1.6 + 0.1j])
    d = _dists(*specs)
    got = gpu.ensemble_adaptive(d, wl, m, MU, 8)
    assert got["panels"].sum() > 32768  # 256 B a record
    part = np.array([0, 1, 5, 102, 250, 251, 498, 499])
    unit = (part[:, None] * wl.size + np.arange(wl.size)).reshape(-1)
    sub = {key: v[..., unit, :] if v.ndim == 3 else v[..., unit] for key, v in got.items()}
    few = _dists(*[specs[k] for k in part])
    _compare(sub, O.ensemble_adaptive(_odist(few), wl, m, mu=MU, greek_order=8))
