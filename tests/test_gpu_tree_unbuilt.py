"""A tree that was never built: forces propagated on it are none, and it builds afterwards like any other."""

from __future__ import annotations

import numpy as np
import pytest

import oracle as O
from gpu_util import consts, lognormal_state

pytestmark = pytest.mark.gpu


def test_propagate_without_a_build():
    import torch

    from dem import _native as N

    n = 300
    pos, r, L = lognormal_state(n, seed=2)
    m, eta, sf = consts()
    ctx = N.Context(n)
    tree = N.Tree(ctx, n, 8 * n)
    F_in = torch.ones((3, n), dtype=torch.float64, device=ctx.device)
    tree.propagate_forces(None)
    tree.propagate_forces(F_in)
    assert ctx.device_errors() == 0 and tree.stats()["node_count"] == 0
    soa = torch.as_tensor(np.ascontiguousarray(pos.T), device=ctx.device)
    F, V = torch.empty_like(soa), torch.empty_like(soa)
    tree.build(n, soa, torch.as_tensor(r, device=ctx.device), L, True, 4)
    tree.forces(m, 0.25, F)
    tree.propagate_forces(None)
    tree.velocity(None, eta, 0.25, sf, V)
    ref = O.Tree(n, 0.5, 4)
    ref.build(pos, r, L, True)
    F_ref, V_ref = ref.forces_and_total_velocity(m, eta, sf)
    np.testing.assert_array_equal(F.cpu().numpy().T, F_ref)
    np.testing.assert_array_equal(V.cpu().numpy().T, V_ref)
