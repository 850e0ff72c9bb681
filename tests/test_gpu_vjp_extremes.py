"""The adjoint's passes (csrc/direct_vjp.cu) with one droplet whose radius or position leaves the range: it takes its
own terms with it (every pair of an infinite radius is cut, a pair too far apart for its squared distance has no
term, a radius of zero has no weight), and the others' are the plain FP64 sums over the pairs that remain."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-10  # norm-wise, as in test_gpu_vjp_blocks.py


def _sums(x, r, F, lam, mu, m, eta, gamma):
    """mu and the gradients of every droplet, open box: the terms of each pair that has them, in plain numpy."""
    n = len(r)
    u, g, s = np.zeros((n, 3)), np.zeros((n, 3)), np.zeros(n)
    for i in range(n):
        with np.errstate(all="ignore"):
            d = x - x[i]
            r2 = (d * d).sum(1)
            have = np.isfinite(r2)
            have[i] = False
            keep = have & (np.sqrt(r2) > r + r[i])
        dist = np.sqrt(r2[have])
        e = d[have] / dist[:, None]
        u[i] = (lam[have] / dist[:, None] + e * ((e * lam[have]).sum(1) / dist)[:, None]).sum(0)
        for a, b in ((np.broadcast_to(lam[i], e.shape), F[have]), (lam[have], np.broadcast_to(F[i], e.shape))):
            ea, eb, ab = (e * a).sum(1), (e * b).sum(1), (a * b).sum(1)
            K = (eb[:, None] * a + ea[:, None] * b - ab[:, None] * e - 3 * (ea * eb)[:, None] * e) / dist[:, None] ** 2
            g[i] -= eta * K.sum(0)
        if not keep.any():
            continue
        dist = np.sqrt(r2[keep])
        e, w, nu = d[keep] / dist[:, None], r[keep] ** 3, mu[keep] - mu[i]
        en, q = (e * nu).sum(1), e[:, 2] ** 2
        H = (15 * q - 3)[:, None] * nu + ((15 - 105 * q) * en + 30 * e[:, 2] * nu[:, 2])[:, None] * e
        H[:, 2] += 30 * e[:, 2] * en - 6 * nu[:, 2]
        g[i] += m / 3 * r[i] ** 3 * (w[:, None] * H / dist[:, None] ** 5).sum(0)
        s[i] = (w * ((5 * q - 1) * en - 2 * e[:, 2] * nu[:, 2]) / dist**4).sum()
    with np.errstate(all="ignore"):
        mu_ref = eta * u + lam / (gamma * r)[:, None]
        gr = -3 * m * r**2 * s - (lam * F).sum(1) / (gamma * r**2)
    return mu_ref, g, gr


@pytest.mark.parametrize("n", [70, 2081])
@pytest.mark.parametrize("case", ["infinite radius", "radius not a number", "radius 1e110", "zero radius", "position 1e200",
                                  "none"])
def test_one_droplet_out_of_range(n, case):
    import torch

    from dem import _native as N

    m, eta, gamma = 2.0, 0.3, 1.7
    rng = np.random.default_rng(n)
    x, F, lam = rng.random((n, 3)), rng.normal(size=(n, 3)), rng.normal(size=(n, 3))
    r = rng.uniform(0.02, 0.1, n) * n ** (-1 / 3)
    k = n - 3
    if case == "position 1e200":
        x[k, 1] = 1e200
    elif case != "none":
        r[k] = {"infinite radius": np.inf, "radius not a number": np.nan, "radius 1e110": 1e110, "zero radius": 0.0}[case]
    if case == "zero radius":
        x[k - 1] = x[k] + 0.3 * r[k - 1]  # in contact with it
    ctx = N.Context(n)

    def dev(a):
        return torch.as_tensor(np.ascontiguousarray(a.T), device=ctx.device)

    mu, g, gr = (torch.empty_like(dev(v)) for v in (x, x, r))
    ctx.direct_vjp(n, dev(x), dev(r), dev(F), dev(lam), m, eta, gamma, 1.0, False, mu, g, gr)
    mu, g, gr = mu.cpu().numpy().T, g.cpu().numpy().T, gr.cpu().numpy()
    mu_ref, g_ref, gr_ref = _sums(x, r, F, lam, np.where(r[:, None] == 0, 0.0, mu), m, eta, gamma)
    rest = np.arange(n) != k if "radius" in case else np.ones(n, bool)
    for a, b in ((mu, mu_ref), (g, g_ref), (gr, gr_ref)):
        assert np.linalg.norm(a[rest] - b[rest]) <= TOL * np.linalg.norm(b[rest])
    if "radius" not in case:  # (the gradients of a radius out of range are infinity times zero)
        assert np.isfinite(g[k]).all()
