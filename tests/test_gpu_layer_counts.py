"""Layered spheres of every kernel's layer counts: 2, 3 and 4 with their state in registers, 5 to 16
in local memory; derivatives of 2 and 3 layers along a direction known at compile time, to 4 and to
16 along any. Values against the oracle (fixed grid and adaptive, 1e-11 as the three-layer tests);
derivatives against the same particle with fewer layers: a layer cut into several of one index has
the sum of their derivatives along its index, keeps its interfaces', and the cuts have none."""

import numpy as np
import pytest

from oracle import oracle as O
from scatrs_b200 import _native
from scatrs_b200 import workloads as W
from test_gpu_adaptive import MU, _compare as _compare_adaptive, _dists, _odist
from test_gpu_ensemble import _compare

pytestmark = pytest.mark.gpu

WL = np.array([0.45, 0.7])


def _particles(n, layers, seed):
    rng = np.random.default_rng(seed)
    fr = np.sort(rng.uniform(0.3, 0.98, (n, layers - 1)), axis=1)
    ml = rng.uniform(1.3, 2.0, (n, layers, 1)) + 1j * rng.choice([0.0, 1e-4, 0.02, 0.2],
                                                                 (n, layers, 1))
    return fr, np.repeat(ml, WL.size, axis=2)


@pytest.mark.parametrize("layers", [2, 4, 5, 16])
def test_fixed_grid_values(gpu, layers):
    d = W.lognormals([0.12, 0.4, 0.9], [1.5, 1.4, 1.3], 3)
    fr, ml = _particles(3, layers, layers)
    got = gpu.ensemble_fixed_layered(d, WL, fr, ml, MU, 70, 12)
    od = np.zeros(3, dtype=O.DIST_DTYPE)
    od["kind"], od["p"], od["r_lo"], od["r_hi"] = d["kind"], d["param"], d["r_lo"], d["r_hi"]
    _compare(got, O.ensemble_fixed_layered(od, WL, fr, ml, 70, MU, 12), tol=1e-11)


@pytest.mark.parametrize("layers", [2, 4, 5, 16])
def test_adaptive_values(gpu, layers):
    d = _dists((1, 0.2, 1.5), (2, 0.3, 0.12), (5, 0.4))
    fr, ml = _particles(3, layers, 10 + layers)
    got = gpu.ensemble_adaptive_layered(d, WL, fr, ml, MU, 12)
    ref = O.ensemble_adaptive_layered(_odist(d), WL, fr, ml, MU, 12)
    _compare_adaptive(got, ref, tol=1e-11)


def _cut(fr, ml, parts):
    """Every layer l cut into parts[l] of its index at equal steps between its interfaces."""
    edge = np.concatenate([np.full((fr.shape[0], 1), 0.2), fr, np.ones((fr.shape[0], 1))], axis=1)
    inner, index = [], []
    for l, k in enumerate(parts):
        index += [l] * k
        for j in range(1, k):
            inner.append(edge[:, l] + (edge[:, l + 1] - edge[:, l]) * j / k)
        if l + 1 < len(parts):
            inner.append(edge[:, l + 1])
    return np.stack(inner, axis=1), ml[:, index], np.array(index)


@pytest.mark.parametrize("parts", [(2, 1), (1, 2, 1), (2, 1, 2), (5, 6, 5)],
                         ids=lambda p: f"{len(p)}-{sum(p)}")
def test_derivatives_of_cut_layers(gpu, parts):
    base = len(parts)
    d = W.lognormals([0.12, 0.3], [1.5, 1.4], 3)
    fr, ml = _particles(2, base, 40)
    frc, mlc, index = _cut(fr, ml, parts)
    got = _native.ensemble_fixed_layered_d(d, WL, frc, mlc, MU, 48, 8)
    want = _native.ensemble_fixed_layered_d(d, WL, fr, ml, MU, 48, 8)
    layers, n_theta = index.size, 2
    cuts = np.flatnonzero(index[:-1] == index[1:])
    kept = np.flatnonzero(index[:-1] != index[1:])
    for k in range(3):
        v, w = got[k], want[k]
        assert np.abs(v - w).max() <= 1e-11 * np.abs(w).max()
        dv, dw = got[3 + k], want[3 + k]
        size = np.abs(dw).reshape(dw.shape[0], -1).max(axis=1)

        def close(a, blk):
            assert np.abs(a - dw[blk]).max() <= 1e-9 * size[blk], (k, blk)

        for p in range(n_theta):
            close(dv[p], p)
        for l in range(base):
            of = np.flatnonzero(index == l)
            for part in range(2):
                close(dv[n_theta + 2 * of + part].sum(axis=0), n_theta + 2 * l + part)
        for j, f in enumerate(kept):
            close(dv[n_theta + 2 * layers + f], n_theta + 2 * base + j)
        for f in cuts:
            assert np.abs(dv[n_theta + 2 * layers + f]).max() <= 1e-9 * size.max()
