"""The Morton-tree walks (csrc/bh.cu) at the edges of their 64-target groups and of the size from which the
groups come from the SMs' queues: theta = 0 (every pair exact) against the same sums in FP64 (pairs closer
than r_i + r_j left out of both, as the walks do), and the same bits in two calls (every group taken once)."""

from __future__ import annotations

import numpy as np
import pytest

from gpu_util import rel_norm

pytestmark = pytest.mark.gpu


def _calc(n, L, periodic, theta):
    from dem.octree import MortonTreeForceCalculator

    return MortonTreeForceCalculator(num_particles=n, theta=theta, mpl=16, eta_oil=0.06, L=L, periodic=periodic)


def _sums(pos, r, F, L, periodic, m, eta):
    out_f, out_v = np.zeros_like(pos), np.zeros_like(pos)
    for i in range(len(r)):
        d = pos - pos[i]
        if periodic:
            d = np.where(np.abs(d) > 0.5 * L, d - np.sign(d) * L, d)
        r2 = (d * d).sum(1)
        keep = r2 >= (r + r[i]) ** 2
        keep[i] = False
        d, r2, rj, f = d[keep], r2[keep], r[keep], F[keep]
        M = m * r[i] ** 3 * rj**3 / r2**3.5
        z2, xy2 = d[:, 2] ** 2, d[:, 0] ** 2 + d[:, 1] ** 2
        out_f[i] = (M * (4 * z2 - xy2)) @ d * [1, 1, 0] + [0, 0, (M * (2 * z2 - 3 * xy2) * d[:, 2]).sum()]
        inv = r2**-0.5
        out_v[i] = eta * ((f * inv[:, None]).sum(0) + ((d * f).sum(1) * inv**3) @ d)
    return out_f, out_v


@pytest.mark.parametrize("periodic", [True, False])
@pytest.mark.parametrize("n", [1, 63, 64, 65, 257, 4097])
def test_exact_walk(n, periodic):
    rng = np.random.default_rng(n)
    L = 3.5e-5 * n ** (1 / 3)
    pos, r = rng.uniform(0, L, (n, 3)), rng.uniform(2e-6, 8e-6, n)
    calc = _calc(n, L, periodic, 0.0)
    F, V = calc.calculate_forces_and_convection(pos, r)
    Fd, Vd = _sums(pos, r, F, L, periodic, calc.m_const, calc.eta_const)
    if n > 1:
        assert rel_norm(F, Fd) <= 1e-5 and rel_norm(V, Vd) <= 2e-5  # FP32 terms; the walk's own bound at theta = 0
    else:
        assert not F.any() and not V.any()


@pytest.mark.parametrize("n", [131071, 131072, 131073, 131136])
def test_queued_groups(n):
    rng = np.random.default_rng(1)
    L = 3.5e-5 * n ** (1 / 3)
    pos, r = rng.uniform(0, L, (n, 3)), rng.uniform(2e-6, 6e-6, n)
    calc = _calc(n, L, True, 0.5)
    first = calc.calculate_forces_and_total_velocity(pos, r, 0.5)
    counts = calc.stats()
    again = calc.calculate_forces_and_total_velocity(pos, r, 0.5)
    assert all(np.array_equal(a, b) for a, b in zip(first, again)) and calc.stats() == counts
    assert all(np.isfinite(a).all() and (np.abs(a).sum(1) > 0).all() for a in first)
