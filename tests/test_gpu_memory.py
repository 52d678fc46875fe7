"""Device memory the library holds: given back by scatrs_release, and sized by the call."""

import numpy as np
import pytest

from scatrs_b200 import _scatrs
from scatrs_b200 import workloads as W

pytestmark = pytest.mark.gpu

MIB = 1 << 20


def _free():
    import torch

    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def _used(lib, call):
    """What a call leaves on the device, from a released library to the next release."""
    lib.scatrs_release()
    before = _free()
    call()
    return before - _free()


def test_release_gives_every_buffer_back(gpu):
    lib = gpu.load()
    mu, wl = W.gauss_legendre(32), np.array([0.5, 0.8])
    m = np.full(2, 1.5 + 1e-2j)

    def calls():
        d = W.lognormals([0.3], [1.5], 3)
        gpu.ensemble_fixed(d, wl, m[None], mu, 64, 16)
        _scatrs.ensemble_compute([(("lognormal", 0.2, 1.5), ("sphere", m), 1.0)], wl, False, 16,
                                 False, mu, True, [], 1e-6, 4096, False, False)
        gpu.spheroid_compute(np.full(4, 12.0), 2.0, 1.5 + 1e-2j, n_terms=24, n_theta=60)

    calls()  # the modules are loaded with their first launches
    lib.scatrs_release()
    before = _free()
    calls()
    held = before - _free()
    lib.scatrs_release()
    assert held > 64 * MIB
    assert before - _free() <= 4 * MIB


@pytest.fixture
def small_arena(gpu):
    """Coefficient arenas of 64 MiB."""
    gpu.set_tuning(arena_rows=1 << 16)
    yield gpu
    gpu.set_tuning()


# The buffers of a call whatever its size, in MiB, at that arena: the coefficient rows, u_k(mx) and
# u_k(x) of the rows and of two more per chunk of the largest slab, and 64 KiB for each of the rest.
FIXED = 64 + (64 + 512) / 2 + (64 + 512) / 4 + 16


def test_a_small_call_holds_little(small_arena):
    gpu = small_arena
    wl, m = np.array([0.5, 0.8]), np.full((1, 2), 1.5 + 1e-2j)
    d = W.lognormals([0.1], [1.4], 3)

    def call():
        gpu.ensemble_fixed_d(d, wl, m, W.gauss_legendre(32), 64, 16)

    call()
    # And the sums of the largest slab's chunks, 5 blocks of 8.
    assert _used(gpu.load(), call) <= (FIXED + 80 + 16) * MIB


def test_a_growth_that_fits_only_exactly(gpu):
    # Regrown buffers take room to spare where there is some: 200 and 200 and 30 MiB, with the room
    # 264, 264 and 45, in 520 MiB.
    import torch

    n_q, n, order = 64, 200 * MIB // (24 * 64), 8
    phase = torch.ones(6, n, n_q, dtype=torch.float64, device="cuda")
    out = torch.empty(6, n, order + 1, dtype=torch.float64, device="cuda")
    gpu.project_greek_device(phase.data_ptr(), 4, n_q, order, 1, out.data_ptr())
    torch.cuda.empty_cache()
    fill = torch.empty(_free() - 520 * MIB, dtype=torch.uint8, device="cuda")
    try:
        gpu.project_greek_device(phase.data_ptr(), n, n_q, order, 1, out.data_ptr())
        torch.cuda.synchronize()
        assert abs(float(out[0, -1, 0]) - 1.0) < 1e-5
    finally:
        del fill
        torch.cuda.empty_cache()
        gpu.load().scatrs_release()


def test_split_chunks_scratch_is_bounded(gpu):
    # 200 chunks of 1,600 orders, few enough for a block each: their scratch is 2 KiB per order, at
    # most half of the arena's bytes. The results have the same bits with and without.
    wl = np.linspace(0.5, 0.501, 200)
    d = W.lognormals([1500 * 0.5 / (2 * np.pi)], [1.01], 1)
    m = np.full((1, 200), 1.33 + 1e-4j)

    def call():
        return gpu.ensemble_fixed(d, wl, m, np.array([-0.5, 0.9]), 32)

    try:
        gpu.set_tuning(arena_rows=1 << 22)
        want = call()
        gpu.set_tuning(arena_rows=1 << 20)
        # The coefficient rows, u_k(mx) and u_k(x) with two rows for each of 2^18 chunks, the sums.
        fixed = 1024 + (1024 + 512) / 2 + (1024 + 512) / 4 + 16
        assert _used(gpu.load(), call) <= (fixed + 64) * MIB
        for a, b in zip(call()[:2], want[:2]):
            assert np.array_equal(a, b)
    finally:
        gpu.set_tuning()
        gpu.load().scatrs_release()


def test_slot_elements_are_bounded(small_arena):
    # 4,000 units of one phase level each at 2,048 cosines: 64 KiB of interpolated elements a unit, a
    # quarter of the arena's bytes at a time.
    gpu = small_arena
    wl = np.linspace(0.5, 0.6, 4000)
    d = W.lognormals([0.1], [1.3], 2)
    m = np.full((1, 4000), 1.5 + 1e-2j)
    mu = W.gauss_legendre(2048)

    def call(sel=slice(None)):
        return gpu.ensemble_fixed(d, wl[sel], m[:, sel], mu, 32)

    phase = 6 * 4000 * 2048 * 8 / MIB
    assert _used(gpu.load(), call) <= (FIXED + phase + 96) * MIB
    got = call()
    for u in (0, 255, 256, 3999):
        one = call(slice(u, u + 1))
        for a, b in zip(got[:2], one[:2]):
            assert np.array_equal(a[:, u], b[:, 0])


def test_kept_level_sets_are_bounded(small_arena):
    # Greek orders in turn, each with its own phase levels (about 500 MiB at these cosines and sizes).
    gpu = small_arena
    lib = gpu.load()
    wl, m = np.array([0.5]), np.array([[1.33 + 1e-4j]])
    d = W.lognormals([900 * 0.5 / (2 * np.pi)], [1.02], 1)
    mu = W.gauss_legendre(4096)

    def call(order):
        return gpu.ensemble_fixed(d, wl, m, mu, 32, order)

    one = _used(lib, lambda: call(4))
    assert one > 256 * MIB
    want = call(6)

    def several():
        for order in range(4, 11):
            call(order)

    # Sets up to 1 GiB together, and the one that is added then.
    assert _used(lib, several) <= one + (1024 + 64) * MIB + one
    for a, b in zip(call(6), want):
        assert np.array_equal(a, b)


def test_bands_are_built_for_the_call_alone(small_arena):
    # No cosines, so projector bands alone: 4 n_q (L + 1) and 2 h ld doubles for each up to the
    # largest chunk's (bands of 1.25 times the last one's terms).
    gpu = small_arena
    wl, m, order = np.array([0.5]), np.array([[1.33 + 1e-4j]]), 2000
    x, n = 800.0, []
    d = W.lognormals([x * wl[0] / (2 * np.pi)], [1.001], 1)
    top = x * 1.001 + 6 * x ** (1 / 3) + 4
    tables, u = 0, 1
    while not n or n[-1] < top:
        k = min(order, 2 * u)
        n_q = u + (k + 2) // 2
        tables += 4 * n_q * (k + 32) * 8 + (n_q + 64) * (u + 16) * 8
        n.append(u)
        u = -(-5 * u // 4)

    def call():
        return gpu.ensemble_fixed(d, wl, m, None, 32, order)

    assert _used(gpu.load(), call) <= (FIXED + 64) * MIB + tables
