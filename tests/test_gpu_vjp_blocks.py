"""The adjoint's block-pair passes (csrc/direct_vjp.cu) at the edges of their blocks (32, 64 and 128
droplets), of the sizes that choose them, and past the size whose records take several launches: sampled
rows against torch autograd of those rows' pair terms in FP64."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-10  # norm-wise; FP64 sums over up to 93,000 terms of both signs


@pytest.mark.parametrize("periodic", [True, False])
@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 1999, 2000, 2001, 4097, 10500, 10501, 32769, 93057])
def test_sampled_rows(n, periodic):
    import torch

    from dem import _native as N

    m, eta, gamma, L = 2.0, 0.3, 1.7, 1.0
    g = torch.Generator("cuda").manual_seed(n)
    kw = dict(device="cuda", dtype=torch.float64, generator=g)
    x, lam = torch.rand((3, n), **kw), torch.randn((3, n), **kw)
    r = (0.05 + 0.2 * torch.rand(n, **kw)) * n ** (-1 / 3)
    ctx = N.Context(n)
    F, mu, gx, gr = (torch.empty_like(v) for v in (x, x, x, r))
    ctx.direct_forces(n, x, r, m, L, periodic, N.PREC_FP64, F)
    ctx.direct_vjp(n, x, r, F, lam, m, eta, gamma, L, periodic, mu, gx, gr)
    assert ctx.device_errors() == 0

    rows = torch.unique(torch.cat([torch.arange(0, min(n, 40)), torch.arange(max(0, n - 40), n)])).cuda()
    xs, rs = x[:, rows].clone().requires_grad_(True), r[rows].clone().requires_grad_(True)
    d = x[:, None, :] - xs[:, :, None]
    if periodic:
        d = torch.where(d.abs() > 0.5 * L, d - torch.sign(d) * L, d)
    other = torch.arange(n, device="cuda")[None, :] != rows[:, None]
    r2 = torch.where(other, (d * d).sum(0), torch.ones_like(d[0]))
    dist = r2.sqrt()
    keep = other & (dist.detach() > r[None, :] + r[rows, None])
    f = torch.stack([(4 * d[2] ** 2 - d[0] ** 2 - d[1] ** 2) * d[0], (4 * d[2] ** 2 - d[0] ** 2 - d[1] ** 2) * d[1],
                     (2 * d[2] ** 2 - 3 * d[0] ** 2 - 3 * d[1] ** 2) * d[2]]) / dist**7
    dipole = m * rs[:, None] ** 3 * r[None, :] ** 3 * ((mu[:, rows, None] - mu[:, None, :]) * f).sum(0)
    zero = torch.zeros_like(r2)

    def oseen(a, b):  # a.G(d) b
        return torch.where(other, (a * b).sum(0) / dist + (a * d).sum(0) * (b * d).sum(0) / dist**3, zero)

    pairs = torch.where(keep, dipole, zero) + eta * (oseen(lam[:, rows, None], F[:, None, :])
                                                     + oseen(F[:, rows, None], lam[:, None, :]))
    total = pairs.sum() + ((lam * F).sum(0)[rows] / (gamma * rs)).sum()
    gx_ref, gr_ref = torch.autograd.grad(total, (xs, rs))
    inv = torch.where(other, 1 / dist, zero).detach()
    dl = (d.detach() * lam[:, None, :]).sum(0) * inv**3
    mu_ref = lam[:, rows] / (gamma * r[rows]) + eta * (lam[:, None, :] * inv + d.detach() * dl).sum(-1)

    def err(a, b):
        return float((a - b).norm()) <= TOL * float(b.norm()) + 1e-300

    assert err(mu[:, rows], mu_ref) and err(gx[:, rows], gx_ref) and err(gr[rows], gr_ref)
