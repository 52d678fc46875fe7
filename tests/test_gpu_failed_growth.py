"""Every device allocation of a call failing in turn, as an out-of-memory cudaMalloc would: the
failed call raises, and the next ones give what an undisturbed library gives."""

import numpy as np
import pytest

from scatrs_b200 import workloads as W
from scatrs_b200.errors import DeviceError

pytestmark = pytest.mark.gpu


def _same(got, want):
    if isinstance(want, dict):
        return set(got) == set(want) and all(_same(got[k], want[k]) for k in want)
    if isinstance(want, (list, tuple)):
        return len(got) == len(want) and all(_same(a, b) for a, b in zip(got, want))
    if want is None or got is None:
        return got is want
    return np.array_equal(got, want)


def _each_growth(lib, small, large, larger=None):
    """`large` with its k-th growth failing, k = 1, 2, ..., in a fresh library and after `small`
    grew it halfway; then `large`, `small` and `larger` again. Returns the number of growths that
    failed."""
    want_small, want_large = small(), large()
    want_larger = larger() if larger else None
    failed = 0
    for first in (None, small):
        k = 0
        while True:
            k += 1
            lib.scatrs_release()
            if first is not None:
                first()
            lib.scatrs_testing_fail_allocation(k)
            try:
                large()
                break
            except DeviceError as e:
                assert "out of memory" in str(e)
            finally:
                lib.scatrs_testing_fail_allocation(0)
            failed += 1
            assert _same(large(), want_large), (k, first is not None)
            assert _same(small(), want_small), (k, first is not None)
            if larger:
                assert _same(larger(), want_larger), (k, first is not None)
    return failed


@pytest.fixture
def small_arena(gpu):
    """Slabs of 64 MiB, so that a fresh library grows quickly."""
    gpu.set_tuning(arena_rows=1 << 16)
    yield gpu
    gpu.set_tuning()


WL = np.array([0.5, 0.7])
M = np.array([[1.5 + 1e-2j, 1.4 + 1e-3j]])
FORMS = {
    # Projector bands alone, on no cosines; phase levels with and without bands beyond them.
    "bands": lambda gpu, d: gpu.ensemble_fixed(d, WL, M, None, 64, 12),
    "levels": lambda gpu, d: gpu.ensemble_fixed(d, WL, M, W.gauss_legendre(90), 64, 12),
    "beyond": lambda gpu, d: gpu.ensemble_fixed(d, WL, M, W.gauss_legendre(4), 64, 12),
    "mixed": lambda gpu, d: gpu.ensemble_fixed(d, WL, M, W.gauss_legendre(60), 64, 12,
                                               i8_above=16),
    "derivatives": lambda gpu, d: gpu.ensemble_fixed_d(d, WL, M, W.gauss_legendre(60), 64, 12),
    "adaptive": lambda gpu, d: gpu.ensemble_adaptive(d, WL, M[0], W.gauss_legendre(20), 12,
                                                     rtol=1e-4),
}


@pytest.mark.parametrize("form", FORMS)
def test_tables(small_arena, form):
    gpu = small_arena

    def call(median):
        return lambda: FORMS[form](gpu, W.lognormals([median], [1.3], 2))

    assert _each_growth(gpu.load(), call(0.1), call(0.8), call(3.0)) >= 10


@pytest.mark.parametrize("precision", [0, 1])
def test_projection(gpu, precision):
    import torch

    def call(n_q, order):
        f = torch.linspace(0.5, 1.5, 6 * 3 * n_q, dtype=torch.float64, device="cuda")
        out = torch.zeros(6, 3, order + 1, dtype=torch.float64, device="cuda")

        def run():
            out.zero_()
            gpu.project_greek_device(f.data_ptr(), 3, n_q, order, precision, out.data_ptr())
            return out.cpu().numpy()

        return run

    assert _each_growth(gpu.load(), call(96, 20), call(128, 40)) >= 6


def test_orientation_average(gpu):
    def call(n):
        return lambda: gpu.spheroid_compute(np.array([1.5, 2.0]), [1.5, 0.6], 1.4 + 1e-2j,
                                            n_terms=n, n_theta=2 * n, greek_order=8)

    # A fresh library: 13 buffers of the T-matrices, 3 of the projection, 10 of the average, the two
    # Clebsch-Gordan tables among them.
    assert _each_growth(gpu.load(), call(6), call(20)) >= 26
