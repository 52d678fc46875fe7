"""The work that users have this framework do, as timed cases through its public entry points.

A case is one call (or one forward and backward pass) on one of these paths:

* ``call``       the fixed grid from host arrays (a script's direct call; small to moderate);
* ``device``     the fixed grid on device arrays (a retrieval's or lookup table's batch), in FP64
                 (``i8_above`` 0) or in the mixed form (above that many terms, int8 digit
                 products);
* ``droplets``   large gamma droplets: phase matrices at thousands of Gauss cosines, then their
                 Greek projection on the tensor cores;
* ``gradient``   a retrieval step on spheres: forward, then backward to the size parameters and
                 the refractive index;
* ``layered``    layered spheres from host arrays; ``layered_gradient`` a retrieval step on them;
* ``adaptive``   the reference's default integration of one distribution; ``adaptive_batch`` of
                 several distributions on shared panels;
* ``spheroids``  randomly oriented spheroids on a fixed grid, every T-matrix converged.

Sizes are those of the benchmark configurations (``scatrs_b200.workloads``), of the tests, or
fractions of them.
"""

from __future__ import annotations

import functools
import math

import numpy as np
import torch

from scatrs_b200 import _native, _scatrs, autograd, ensemble_fixed, gauss_legendre
from scatrs_b200.workloads import gammas, lognormals

SCALARS = 11


def listed():
    return [
        # One lognormal at three wavelengths: a script's or a notebook's call.
        dict(name="call_small", path="call", kind="lognormal", n_dist=1, n_wl=3, n_nodes=256,
             n_mu=180, order=32),
        # A few gamma distributions over a spectrum, odd sizes everywhere, copies included.
        dict(name="call_ragged", path="call", kind="gamma", n_dist=5, n_wl=33, n_nodes=301,
             n_mu=181, order=50),
        # A moderate lookup table on the device in FP64.
        dict(name="device_table", path="device", n_dist=16, n_wl=128, n_nodes=512, n_mu=360,
             order=64, i8_above=0),
        # Half of the batched configuration in FP64.
        dict(name="device_batch", path="device", n_dist=64, n_wl=512, n_nodes=512, n_mu=360,
             order=64, i8_above=0),
        # The whole batched configuration in the mixed form.
        dict(name="device_mixed", path="device", n_dist=64, n_wl=1024, n_nodes=512, n_mu=360,
             order=64, i8_above=48),
        # Cloud droplets: size parameters to a thousand, phase matrices at 4096 Gauss cosines.
        dict(name="droplets", path="droplets", n_dist=6, n_wl=16, n_nodes=256, n_mu=4096,
             order=1024),
        # A retrieval step (forward and backward).
        dict(name="gradient", path="gradient", n_dist=16, n_wl=48, n_nodes=256, n_mu=180,
             order=32),
        # Coated particles, values only.
        dict(name="layered", path="layered", n_dist=24, n_wl=64, n_nodes=256, n_mu=180, order=32),
        # A retrieval step on three-layer spheres.
        dict(name="layered_gradient", path="layered_gradient", n_dist=16, n_wl=48, n_nodes=256,
             n_mu=180, order=32),
        # The reference's default call: one distribution, a short spectrum, Greek coefficients.
        dict(name="adaptive", path="adaptive", n_dist=1, n_wl=24, n_mu=0, order=64),
        # Sixteen distributions over a spectrum on shared panels.
        dict(name="adaptive_batch", path="adaptive_batch", n_dist=16, n_wl=64, n_mu=181,
             order=64),
        # Dust-like spheroids at the workload's aspect ratios, a few sizes each.
        dict(name="spheroids", path="spheroids", n_dist=8, n_wl=1, n_nodes=36, n_mu=180,
             order=64),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(["call", "device", "device", "droplets", "gradient", "layered",
                       "layered_gradient", "adaptive", "adaptive_batch", "spheroids"])
    c = dict(path=path, n_mu=rng.choice([91, 180, 181, 360]), order=rng.randint(16, 64))
    if path == "call":
        c.update(kind=rng.choice(["lognormal", "gamma"]), n_dist=_log(rng, 1, 8),
                 n_wl=_log(rng, 1, 64), n_nodes=rng.randint(64, 512))
    elif path == "device":
        c.update(n_dist=_log(rng, 2, 64), n_wl=_log(rng, 8, 256), n_nodes=rng.randint(200, 512),
                 i8_above=rng.choice([0, 32, 48]))
    elif path == "droplets":
        c.update(n_dist=rng.randint(1, 6), n_wl=rng.randint(2, 16), n_nodes=256,
                 n_mu=rng.choice([2048, 4096]), order=rng.choice([512, 1000, 1024]))
    elif path in ("gradient", "layered_gradient"):
        c.update(n_dist=_log(rng, 1, 16), n_wl=_log(rng, 4, 48), n_nodes=rng.randint(100, 256))
    elif path == "layered":
        c.update(n_dist=_log(rng, 1, 24), n_wl=_log(rng, 4, 64), n_nodes=rng.randint(100, 256))
    elif path == "adaptive":
        c.update(n_dist=1, n_wl=_log(rng, 1, 64), n_mu=rng.choice([0, 91]))
    elif path == "adaptive_batch":
        c.update(n_dist=rng.randint(2, 16), n_wl=_log(rng, 4, 64))
    else:
        c.update(n_dist=rng.randint(1, 8), n_wl=1, n_nodes=rng.randint(16, 36))
    return c


def _spread(rng, lo, hi, n, log=False):
    """n values stratified over [lo, hi], so that every seed has the same range of sizes."""
    u = (rng.permutation(n) + rng.uniform(0.25, 0.75, n)) / n
    return np.exp(np.log(lo) + u * np.log(hi / lo)) if log else lo + u * (hi - lo)


def _inputs(case, seed):
    """The distributions, wavelengths and particles of a case, as numpy arrays."""
    rng = np.random.default_rng([int(seed), 7])
    path, nd, nw = case["path"], case["n_dist"], case["n_wl"]
    s = {}
    if path == "call":
        s["wl"] = np.array([0.35, 0.55, 1.0]) if nw == 3 else np.geomspace(0.35, 1.6, nw)
        if case["kind"] == "lognormal":
            s["dists"] = lognormals(_spread(rng, 0.06, 0.3, nd, True), _spread(rng, 1.4, 1.7, nd), 5)
        else:
            s["dists"] = gammas(_spread(rng, 0.2, 2.0, nd, True), _spread(rng, 0.05, 0.2, nd))
        k = np.exp(rng.uniform(np.log(1e-8), np.log(1e-2), (nd, nw)))
        s["m"] = rng.uniform(1.33, 1.60, (nd, 1)) + 1j * k
    elif path == "device":
        s["wl"] = np.geomspace(0.3, 2.5, nw)
        s["dists"] = lognormals(_spread(rng, 0.05, 5.0, nd, True), rng.uniform(1.2, 2.2, nd), 4)
        k = np.exp(rng.uniform(np.log(1e-8), np.log(1e-1), (nd, nw)))
        s["m"] = rng.uniform(1.33, 1.60, (nd, nw)) + 1j * k
    elif path == "droplets":
        s["wl"] = np.geomspace(0.4, 2.2, nw)
        s["dists"] = gammas(_spread(rng, 5.0, 20.0, nd), _spread(rng, 0.05, 0.2, nd))
        s["m"] = 1.33 + 1j * np.exp(rng.uniform(np.log(1e-9), np.log(1e-3), (nd, nw)))
    elif path == "gradient":
        s["wl"] = np.geomspace(0.35, 1.6, nw)
        s["dists"] = lognormals(_spread(rng, 0.05, 1.0, nd), _spread(rng, 1.3, 2.0, nd), 4)
        k = np.exp(rng.uniform(np.log(1e-6), np.log(1e-1), (nd, nw)))
        s["m"] = rng.uniform(1.33, 1.60, (nd, nw)) + 1j * k
    elif path in ("layered", "layered_gradient"):
        s["wl"] = np.geomspace(0.3, 1.6, nw)
        s["dists"] = lognormals(_spread(rng, 0.05, 1.0, nd), _spread(rng, 1.3, 2.0, nd), 4)
        s["fractions"] = np.stack([rng.uniform(0.3, 0.9, nd), rng.uniform(0.9, 0.99, nd)], axis=1)
        k = np.exp(rng.uniform(np.log(1e-6), np.log(0.5), (nd, 3)))
        ml = rng.uniform(1.3, 2.0, (nd, 3)) + 1j * k
        s["m"] = np.ascontiguousarray(np.repeat(ml[:, :, None], nw, axis=2))
    elif path in ("adaptive", "adaptive_batch"):
        s["wl"] = np.geomspace(0.35, 1.6, nw)
        med = _spread(rng, 0.05, 0.5, nd, True)
        s["specs"] = [("lognormal", float(a), float(b))
                      for a, b in zip(med, _spread(rng, 1.3, 1.7, nd))]
        s["m"] = np.full(nw, rng.uniform(1.40, 1.55) + 1j * rng.uniform(1e-3, 1e-2))
    else:  # spheroids: the aspect ratios of the workload, sizes to x = 21
        s["wl"] = np.array([0.55]) if nw == 1 else np.geomspace(0.35, 1.0, nw)
        eps = np.geomspace(0.4, 3.0, nd) if nd > 1 else np.array([0.6])
        med, wid = _spread(rng, 0.2, 1.5, nd), rng.uniform(1.5, 2.0, nd)
        d = lognormals(med, wid, 2)
        d["r_hi"] = np.minimum(d["r_hi"], 21.0 * s["wl"].min() / (2 * np.pi))
        d["r_lo"] = np.minimum(d["r_lo"], d["r_hi"] / 4)
        s["dists"], s["eps"] = d, eps
        k = np.exp(rng.uniform(np.log(1e-4), np.log(1e-1), nd))
        s["m"] = np.repeat((1.53 + 1j * k)[:, None], nw, axis=1)
    return s


def _upstream(case, seed, n, device):
    """The gradients a loss on the scalars, the phase matrix and the Greek coefficients sends."""
    g = torch.Generator().manual_seed(int(seed) * 3 + 1)
    shapes = ((SCALARS, n), (6, n, case["n_mu"]), (6, n, case["order"] + 1))
    return [torch.randn(s, generator=g, dtype=torch.float64).to(device) for s in shapes]


def prepare(case, seed):
    s = _inputs(case, seed)
    s["case"] = case
    path, n_mu, order = case["path"], case["n_mu"], case["order"]
    s["mu"] = gauss_legendre(n_mu)[0] if n_mu else None
    n = case["n_dist"] * case["n_wl"]
    f64 = dict(dtype=torch.float64, device="cuda")
    if path in ("device", "droplets"):
        s["wl_d"] = torch.as_tensor(s["wl"], **f64)
        s["m_d"] = torch.view_as_real(torch.as_tensor(s["m"], device="cuda")).contiguous()
        s["values"] = torch.empty(SCALARS, n, **f64)
        s["phase"] = torch.empty(6, n, n_mu, **f64)
        s["greek"] = torch.empty(6, n, order + 1, **f64)
    elif path in ("gradient", "layered_gradient"):
        s["ranges"] = np.stack([s["dists"]["r_lo"], s["dists"]["r_hi"]], axis=1)
        s["theta"] = torch.as_tensor(np.array(s["dists"]["param"][:, :2]), **f64)
        s["m_re"] = torch.as_tensor(s["m"].real.copy(), **f64)
        s["m_im"] = torch.as_tensor(s["m"].imag.copy(), **f64)
        s["up"] = _upstream(case, seed, n, "cuda")
        if path == "layered_gradient":
            s["frac"] = torch.as_tensor(s["fractions"], **f64)
    return s


def _leaf(t):
    return t.detach().clone().requires_grad_(True)


def run(state):
    s = state
    case, path = s["case"], s["case"]["path"]
    order = case["order"]
    if path == "call":
        return ensemble_fixed(s["dists"], s["wl"], s["m"], s["mu"], case["n_nodes"], order)
    if path in ("device", "droplets"):
        stream = torch.cuda.current_stream().cuda_stream
        droplets = path == "droplets"
        _native.ensemble_fixed_device(s["dists"], s["wl_d"].data_ptr(), case["n_wl"],
                                      s["m_d"].data_ptr(), s["mu"], case["n_nodes"],
                                      -1 if droplets else order, True, s["values"].data_ptr(),
                                      s["phase"].data_ptr(),
                                      0 if droplets else s["greek"].data_ptr(), stream,
                                      i8_above=case.get("i8_above", 0))
        if droplets:
            _native.project_greek_device(s["phase"].data_ptr(), case["n_dist"] * case["n_wl"],
                                         case["n_mu"], order, 1, s["greek"].data_ptr(), stream)
        return s["values"], s["phase"], s["greek"]
    if path in ("gradient", "layered_gradient"):
        args = dict(kind="lognormal", ranges=s["ranges"], wavelengths=s["wl"], mu=s["mu"],
                    n_nodes=case["n_nodes"], greek_order=order)
        leaves = [_leaf(s["theta"]), _leaf(s["m_re"]), _leaf(s["m_im"])]
        if path == "gradient":
            out = autograd.ensemble_fixed(*leaves, **args)
        else:
            leaves.insert(1, _leaf(s["frac"]))
            out = autograd.ensemble_fixed_layered(*leaves, **args)
        torch.autograd.backward(out, s["up"])
        return [t.detach() for t in out], [t.grad for t in leaves]
    if path == "layered":
        return _native.ensemble_fixed_layered(s["dists"], s["wl"], s["fractions"], s["m"],
                                              s["mu"], case["n_nodes"], order)
    if path == "adaptive":
        return _scatrs.ensemble_compute([(s["specs"][0], ("sphere", s["m"]), 1.0)], s["wl"],
                                        False, order, False, s["mu"], True, [], 1e-6, 4096,
                                        False, False)
    if path == "adaptive_batch":
        return _scatrs.ensemble_compute_batch(s["specs"], ("sphere", s["m"]), s["wl"], order,
                                              False, s["mu"], True, 1e-6, 4096, False, False)
    return _native.ensemble_fixed_spheroid(s["dists"], s["wl"], s["eps"], s["m"], s["mu"],
                                           case["n_nodes"], order)


# ---------------------------------------------------------------------------------------------
# The work of a pass: inputs and outputs once, and the operations of the least arithmetic that
# gives them (the recurrences per order, the angle sums, the projections).
# ---------------------------------------------------------------------------------------------
RECURRENCE_FLOPS = 200  # per order and node: the ratios, a_n, b_n and the sums


def _terms(x):
    return np.ceil(x + 6.0 * np.cbrt(x) + 3.0)


def work(case):
    s = _inputs(case, 0)
    path, n_mu, order = case["path"], case["n_mu"], case["order"]
    n = case["n_dist"] * case["n_wl"]
    greek = 6 * n * (order + 1)
    outputs = SCALARS * n + 6 * n * n_mu + greek
    if path in ("adaptive", "adaptive_batch"):
        nodes = 15 * 8  # GK15 nodes of the panels a smooth distribution needs
        lo = np.array([a * b ** -4 for _, a, b in s["specs"]])
        hi = np.array([a * b ** 6 for _, a, b in s["specs"]])
        outputs = 2 * outputs
    else:
        nodes = case["n_nodes"]
        lo, hi = np.array(s["dists"]["r_lo"]), np.array(s["dists"]["r_hi"])
    t = (np.arange(nodes) + 0.5) / nodes
    r = lo[:, None] * (hi / lo)[:, None] ** t[None, :]
    terms = _terms(2 * np.pi * r[:, None, :] / s["wl"][None, :, None])
    # Angle sums: two real sums per non-negative cosine and complex coefficient pair, at the
    # requested cosines and (with Greek coefficients) at terms + (order + 1) / 2 Gauss cosines.
    half = (n_mu + 1) // 2
    project = 0 if path == "droplets" else 0.5 * (terms + 0.5 * (order + 1))
    flops = float((RECURRENCE_FLOPS * terms + 16 * terms * (half + project)).sum())
    if path == "droplets":
        flops += 12.0 * n * n_mu * (order + 1)
    layers = 3 if path.startswith("layered") else 1
    if layers > 1:
        flops += float((2 * RECURRENCE_FLOPS * 4 * terms).sum())
    if path.endswith("gradient"):
        blocks = 2 + 2 * layers + (layers - 1)
        flops *= 1 + 2 * layers if layers > 1 else 2
        outputs *= 1 + blocks
    if path == "spheroids":
        # Per node and mode: 8 surface integrals of terms^2 / 2 pairs over 2 terms nodes, and a
        # solve of 2 terms complex unknowns; the orientation average as many again.
        flops = float((terms * (8 * 8 * terms ** 3 + 8 / 3 * (2 * terms) ** 3 * 4 / 2)).sum())
    inputs = 2 * n * layers + 4 * case["n_dist"] + case["n_wl"] + n_mu
    return {"bytes": 8.0 * (inputs + outputs), "flops": flops}


# ---------------------------------------------------------------------------------------------
# The same outputs from the textbook series in torch, complex128.
# ---------------------------------------------------------------------------------------------
NODE_LIMIT = 1_200_000  # nodes a reference evaluation takes in about ten seconds
DEVICE = "cuda" if torch.cuda.is_available() else "cpu"


@functools.lru_cache(maxsize=None)
def _gauss(n):
    """Gauss-Legendre nodes (ascending) and weights by Newton's method."""
    k = np.arange(1, (n + 1) // 2 + 1)
    x = np.cos(np.pi * (k - 0.25) / (n + 0.5))
    for _ in range(100):
        p0, p1 = np.ones_like(x), x.copy()
        for j in range(2, n + 1):
            p0, p1 = p1, ((2 * j - 1) * x * p1 - (j - 1) * p0) / j
        if n == 1:
            p0, p1 = np.ones_like(x), x.copy()
        dp = n * (x * p1 - p0) / (x * x - 1.0)
        dx = p1 / dp
        x = x - dx
        if np.max(np.abs(dx)) < 4e-16:
            break
    if n % 2:
        x[-1] = 0.0
    w = 2.0 / ((1.0 - x * x) * dp * dp)
    half = n // 2
    return (np.concatenate([-x[:half], x[::-1]]), np.concatenate([w[:half], w[::-1]]))


def _angles(n_max, mu):
    """pi_n and tau_n scaled by (2n + 1) / (n (n + 1)), n = 1..n_max, at the cosines mu."""
    pi_prev, pi = torch.zeros_like(mu), torch.ones_like(mu)
    ps, ts = [], []
    for n in range(1, n_max + 1):
        f = (2 * n + 1) / (n * (n + 1))
        ps.append(f * pi)
        ts.append(f * (n * mu * pi - (n + 1) * pi_prev))
        pi_prev, pi = pi, ((2 * n + 1) * mu * pi - (n + 1) * pi_prev) / n
    return torch.stack(ps), torch.stack(ts)


def _wigner(order, mu):
    """d^l_00, d^l_22, d^l_2-2 and d^l_02 at the cosines mu, l = 0..order, in l's recurrence."""
    out = []
    for a, b in ((0, 0), (2, 2), (2, -2), (0, 2)):
        lo = max(abs(a), abs(b))
        start = {(0, 0): torch.ones_like(mu), (2, 2): 0.25 * (1 + mu) ** 2,
                 (2, -2): 0.25 * (1 - mu) ** 2,
                 (0, 2): math.sqrt(6.0) / 4.0 * (1 - mu * mu)}[(a, b)]
        rows = [torch.zeros_like(mu)] * lo + [start]
        prev, cur = torch.zeros_like(mu), start
        for l in range(lo, order):
            c0 = math.sqrt((l * l - a * a) * (l * l - b * b)) * (l + 1)
            c2 = l * math.sqrt(((l + 1) ** 2 - a * a) * ((l + 1) ** 2 - b * b))
            c1 = (2 * l + 1) * (l * (l + 1) * mu - a * b)
            nxt = mu * cur if l == 0 else (c1 * cur - c0 * prev) / c2
            prev, cur = cur, nxt
            rows.append(cur)
        out.append(torch.stack(rows[: order + 1], dim=1))
    return out


def _log_derivative(z, n):
    """D_k(z) = psi_k'(z) / psi_k(z), k = 0..n, by downward recurrence from far above."""
    size = float(z.detach().abs().max())
    start = int(max(n, size) + 60 + 4.0 * size ** (1 / 3))
    d, out = torch.zeros_like(z), [None] * (n + 1)
    for k in range(start, 0, -1):
        if k <= n:
            out[k] = d
        d = k / z - 1.0 / (d + k / z)
    out[0] = d
    return out


def _outer(z, d1, n):
    """psi_k zeta_k and D3_k(z) = zeta_k' / zeta_k, k = 0..n, upward."""
    e = torch.exp(2j * z)
    pz, d3 = [0.5 * (1.0 - e)], [torch.full_like(z, 1j)]
    for k in range(1, n + 1):
        pz.append(pz[-1] * (k / z - d1[k - 1]) * (k / z - d3[-1]))
        d3.append(d1[k] + 1j / pz[-1])
    return d3


def _coefficients(x, ms, fr):
    """a_n, b_n (n = 1..N of the largest x, zero above each node's own N) of spheres of layers
    with indices ms (innermost first) and outer radii fr (the last 1) over the particle's."""
    n = int(_terms(float(x.max())))
    terms = torch.as_tensor(_terms(x.cpu().numpy()), device=x.device)
    z = ms[0] * fr[0] * x
    ha = _log_derivative(z, n)
    hb = ha
    for l in range(1, len(ms)):
        z1, z2 = ms[l] * fr[l - 1] * x, ms[l] * fr[l] * x
        d1i, d1o = _log_derivative(z1, n), _log_derivative(z2, n)
        d3i, d3o = _outer(z1, d1i, n), _outer(z2, d1o, n)
        e1, e2 = torch.exp(2j * z1), torch.exp(2j * z2)
        q = (1.0 - e1) / (1.0 - e2) * torch.exp(2j * (z2 - z1))  # psi/zeta at z1 over at z2
        na, nb = [None], [None]
        for k in range(1, n + 1):
            q = (q * (k / z1 - d1i[k - 1]) * (k / z2 - d3o[k - 1])
                 / ((k / z2 - d1o[k - 1]) * (k / z1 - d3i[k - 1])))
            g1, g2 = ms[l] * ha[k] - ms[l - 1] * d1i[k], ms[l] * ha[k] - ms[l - 1] * d3i[k]
            na.append((g2 * d1o[k] - q * g1 * d3o[k]) / (g2 - q * g1))
            g1, g2 = ms[l - 1] * hb[k] - ms[l] * d1i[k], ms[l - 1] * hb[k] - ms[l] * d3i[k]
            nb.append((g2 * d1o[k] - q * g1 * d3o[k]) / (g2 - q * g1))
        ha, hb = na, nb
    # psi upward while k <= x, by ratios from above beyond; chi upward.
    ratio = [None] * (n + 2)
    r = torch.zeros_like(x)
    for k in range(int(n + 60 + 4.0 * float(x.max()) ** (1 / 3)), 0, -1):
        r = 1.0 / ((2 * k + 1) / x - r)
        if k <= n:
            ratio[k] = r
    psi_prev, psi = torch.cos(x), torch.sin(x)
    chi_prev, chi = -torch.sin(x), torch.cos(x)
    m_out = ms[-1]
    aa, bb = [], []
    for k in range(1, n + 1):
        up = (2 * k - 1) / x * psi - psi_prev
        psi_prev, psi = psi, torch.where(x >= k, up, psi * ratio[k])
        chi_prev, chi = chi, (2 * k - 1) / x * chi - chi_prev
        xi, xi_prev = torch.complex(psi, -chi), torch.complex(psi_prev, -chi_prev)
        ta, tb = ha[k] / m_out + k / x, hb[k] * m_out + k / x
        on = (terms >= k).to(torch.float64)
        # Beyond a node's own N chi overflows; those orders are dropped.
        a = (ta * psi - psi_prev) / torch.where(terms >= k, ta * xi - xi_prev, 1.0)
        b = (tb * psi - psi_prev) / torch.where(terms >= k, tb * xi - xi_prev, 1.0)
        aa.append(a * on)
        bb.append(b * on)
    return torch.stack(aa), torch.stack(bb)


def _elements(a, b, angles):
    pi, tau = (t.to(torch.complex128) for t in angles)
    s1 = a.transpose(0, 1) @ pi + b.transpose(0, 1) @ tau
    s2 = a.transpose(0, 1) @ tau + b.transpose(0, 1) @ pi
    n1, n2, c = s1.real ** 2 + s1.imag ** 2, s2.real ** 2 + s2.imag ** 2, s2 * s1.conj()
    return torch.stack([0.5 * (n1 + n2), 0.5 * (n2 - n1), c.real, c.imag])


def _density(kind, theta, r):
    """u(r) of a distribution up to a factor, which the averages drop."""
    if kind == "lognormal":
        return torch.exp(-0.5 * (torch.log(r / theta[:, :1]) / torch.log(theta[:, 1:2])) ** 2) / r
    a, b = theta[:, :1], theta[:, 1:2]
    return torch.exp((1.0 - 3.0 * b) / b * torch.log(r / a) - r / (a * b))


def _sums(case, s, theta, ms, fr, adjoint=None):
    """Each unit's weighted sums: 8 per-particle quantities, the four phase elements at the
    requested cosines and the raw Greek projections. With `adjoint` (the gradient along the
    sums) it runs chunk by chunk backward instead."""
    nd, nw, nq = case["n_dist"], case["n_wl"], case["n_nodes"]
    order, n_mu = case["order"], case["n_mu"]
    f64 = dict(dtype=torch.float64, device=DEVICE)
    t, gw = _gauss(nq)
    lo = np.log(np.array(s["dists"]["r_lo"]))[:, None]
    hi = np.log(np.array(s["dists"]["r_hi"]))[:, None]
    r_np = np.exp(0.5 * (hi - lo) * t[None, :] + 0.5 * (hi + lo))
    r = torch.as_tensor(r_np, **f64)
    gw = torch.as_tensor(0.5 * (hi - lo) * gw[None, :], **f64)
    wl = torch.as_tensor(s["wl"], **f64)
    unit = torch.arange(nd * nw, device=DEVICE).repeat_interleave(nq)
    node = torch.arange(nq, device=DEVICE).repeat(nd * nw)
    d, i = unit // nw, unit % nw
    x_all = 2 * math.pi * r[d, node] / wl[i]
    rank = torch.argsort(x_all, descending=True)
    scal = torch.zeros(8, nd * nw, **f64)
    phase = torch.zeros(4, nd * nw, n_mu, **f64)
    greek = torch.zeros(6, nd * nw, order + 1, **f64)
    want_greek = case["path"] != "droplets"
    kind = case.get("kind", "lognormal" if want_greek else "gamma")
    mu = torch.as_tensor(_gauss(n_mu)[0], **f64)
    at = 0
    while at < rank.numel():
        n = int(_terms(float(x_all[rank[at]])))
        rows = max(n_mu, 2 * n)
        size = int(min(1 << 15, max(256, (1 << 29) // (16 * 8 * rows))))
        if adjoint is not None:
            size = min(size, max(256, (1 << 34) // (n * 16 * 150 * len(ms))))
        sel = rank[at:at + size]
        at += size
        ud, ui, u = d[sel], i[sel], unit[sel]
        x, rr = x_all[sel], r[ud, node[sel]]
        with torch.set_grad_enabled(adjoint is not None):
            w = gw[ud, node[sel]] * rr * _density(kind, theta[ud], rr[:, None])[:, 0]
            a, b = _coefficients(x, [m[ud, ui] for m in ms],
                                 [fr[ud, l] for l in range(len(ms) - 1)] + [torch.ones_like(x)])
            k = torch.arange(1, a.shape[0] + 1, **f64)[:, None]
            sca = ((2 * k + 1) * (a.abs() ** 2 + b.abs() ** 2)).sum(0)
            ext = ((2 * k + 1) * (a + b).real).sum(0)
            g = ((k * (k + 2) / (k + 1))[:-1] * (a[:-1] * a[1:].conj()
                                                + b[:-1] * b[1:].conj()).real).sum(0)
            g = g + ((2 * k + 1) / (k * (k + 1)) * (a * b.conj()).real).sum(0)
            back = ((2 * k + 1) * (1 - 2 * (k % 2)) * (a - b)).sum(0)
            area, x2 = math.pi * rr * rr, x * x
            q = torch.stack([torch.ones_like(x), area * 2 / x2 * ext, area * 2 / x2 * sca,
                             area * 4 / x2 * g, area * 2 / x2 * (ext - sca),
                             area * back.abs() ** 2 / x2, rr ** 2, rr ** 3]) * w
            e = _elements(a, b, _angles(a.shape[0], mu)) * (w * 4 / x2 * area)[None, :, None]
            gr = None
            if want_greek:
                cq, cw = (torch.as_tensor(v, **f64) for v in _gauss(a.shape[0] + (order + 2) // 2))
                f = _elements(a, b, _angles(a.shape[0], cq)) * (w * 4 / x2 * area)[None, :, None]
                scale = (2 * torch.arange(order + 1, **f64) + 1) / 2
                d00, d22, d2m2, d02 = (v * cw[:, None] * scale for v in _wigner(order, cq))
                p, mi = (f[0] + f[2]) @ d22, (f[0] - f[2]) @ d2m2
                gr = torch.stack([f[0] @ d00, 0.5 * (p + mi), 0.5 * (p - mi), f[2] @ d00,
                                  f[1] @ d02, f[3] @ d02])
            if adjoint is not None:
                ga, gp, gg = adjoint
                loss = (ga[:, u] * q).sum() + (gp[:, u] * e).sum()
                if gr is not None:
                    loss = loss + (gg[:, u] * gr).sum()
                loss.backward()
                continue
        scal.index_add_(1, u, q)
        phase.index_add_(1, u, e)
        if gr is not None:
            greek.index_add_(1, u, gr)
    return scal, phase, greek


def _assemble(sums):
    """The outputs from the sums: averages, ratios and the normalized phase matrix."""
    scal, phase, greek = sums
    v = scal / scal[0]
    ext, sca, g, ab, back, r2, r3 = v[1:8]
    values = torch.stack([ext, sca, ab, back, sca / ext, g / sca, 4 * math.pi * ext / back,
                          torch.zeros_like(ext), r3 / r2, math.pi * r2, 4 * math.pi / 3 * r3])
    f = phase / scal[0][None, :, None] / sca[None, :, None]
    return values, torch.stack([f[0], f[1], f[0], f[2], f[3], f[2]]), greek / greek[0, :, :1]


def exact(case, seed):
    path = case["path"]
    if path not in ("call", "device", "droplets", "gradient", "layered", "layered_gradient"):
        return None  # adaptive panels and double-double T-matrices: no short statement
    if case["n_dist"] * case["n_wl"] * case["n_nodes"] > NODE_LIMIT:
        return None
    s = _inputs(case, seed)
    layered = path.startswith("layered")
    f64 = dict(dtype=torch.float64, device=DEVICE)
    theta = torch.as_tensor(np.array(s["dists"]["param"][:, :2]), **f64)
    m = torch.as_tensor(s["m"], device=DEVICE)
    re, im = m.real.clone(), m.imag.clone()
    fr = torch.as_tensor(s["fractions"], **f64) if layered else torch.zeros(case["n_dist"], 0,
                                                                           **f64)
    gradient = path.endswith("gradient")
    leaves = [theta, fr, re, im]
    if gradient:
        leaves = [t.requires_grad_(True) for t in leaves]

    def layers():
        m = torch.complex(re, im)
        return [m[:, l] for l in range(m.shape[1])] if layered else [m]

    with torch.no_grad():
        sums = _sums(case, s, theta, layers(), fr)
    if path == "droplets":
        values, phase, _ = _assemble((sums[0], sums[1], torch.ones_like(sums[2])))
        cq, cw = (torch.as_tensor(v, **f64) for v in _gauss(case["n_mu"]))
        scale = (2 * torch.arange(case["order"] + 1, **f64) + 1) / 2
        d00, d22, d2m2, d02 = (v * cw[:, None] * scale for v in _wigner(case["order"], cq))
        p, mi = (phase[0] + phase[3]) @ d22, (phase[0] - phase[3]) @ d2m2
        greek = torch.stack([phase[0] @ d00, 0.5 * (p + mi), 0.5 * (p - mi), phase[3] @ d00,
                             phase[1] @ d02, phase[4] @ d02])
        return values, phase, greek
    if not gradient:
        return _assemble(sums)
    parts = [t.detach().requires_grad_(True) for t in sums]
    out = _assemble(parts)
    n = case["n_dist"] * case["n_wl"]
    torch.autograd.backward(out, _upstream(case, seed, n, DEVICE))
    adjoint = [t.grad for t in parts]
    # The chunks' backward passes share the leaves only.
    _chunked(case, s, theta, layers, fr, adjoint)
    grads = [theta.grad, fr.grad, re.grad, im.grad] if layered else [theta.grad, re.grad, im.grad]
    return [t.detach() for t in out], grads


def _chunked(case, s, theta, layers, fr, adjoint):
    """The backward pass over every chunk: each index leaf is split off once, its gradient
    returned to the real and imaginary parts at the end."""
    ms = [m.detach().requires_grad_(True) for m in layers()]
    _sums(case, s, theta, ms, fr, adjoint)
    torch.autograd.backward(layers(), [m.grad for m in ms])
