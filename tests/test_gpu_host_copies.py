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


def test_managed_outputs(gpu):
    # Memory that the runtime manages is left to its own copy, whatever the size.
    import ctypes

    from scatrs_b200._native import FixedOptions, _p

    import torch

    n, n_mu = 400, 64  # 1.2 MB of phase matrix
    d, wl = W.lognormals(np.full(n, 0.1), 1.4, 2), np.array([0.6])
    m, mu = np.full((n, 1), 1.4 + 0.01j), W.gauss_legendre(n_mu)
    want = _native.ensemble_fixed(d, wl, m, mu, 8)[:2]
    cudart = ctypes.CDLL(None if hasattr(ctypes.CDLL(None), "cudaMallocManaged") else
                         next(p.split()[-1] for p in open("/proc/self/maps")
                              if "libcudart" in p))
    torch.cuda.init()
    got = []
    for a in want:
        p = ctypes.c_void_p()
        assert cudart.cudaMallocManaged(ctypes.byref(p), ctypes.c_size_t(a.nbytes), 1) == 0
        got.append((p, np.ctypeslib.as_array((ctypes.c_double * a.size).from_address(p.value))))
    err = ctypes.create_string_buffer(512)
    opts = FixedOptions(8, -1, 1, 0)
    st = gpu.load().scatrs_ensemble_fixed(
        d.ctypes.data, n, _p(wl), 1, _p(m.view(np.float64).reshape(-1)), _p(mu), n_mu,
        ctypes.byref(opts), ctypes.cast(got[0][0], ctypes.POINTER(ctypes.c_double)),
        ctypes.cast(got[1][0], ctypes.POINTER(ctypes.c_double)), None, err, 512)
    assert st == 0, err.value
    for (p, a), b in zip(got, want):
        assert np.array_equal(a, b.reshape(-1))
        cudart.cudaFree(p)
