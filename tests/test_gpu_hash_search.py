"""The collision search's own grid (csrc/hash.cu) where its choices can go wrong -- radii over orders of
magnitude, one giant droplet, clusters, zero and negative radii, coincident droplets, positions outside the
box, few cells per axis, more pairs than its list holds, a short pair buffer: the oracle's pair sets."""

from __future__ import annotations

import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu

L = 1e-3


def _state(case, n=4000):
    rng = np.random.default_rng(len(case))
    pos, r = rng.uniform(0, L, (n, 3)), rng.uniform(3e-6, 9e-6, n)
    if case == "wide radii":
        r = np.minimum(1e-7 * np.exp(2.0 * rng.standard_normal(n)), 3e-5)
    elif case == "one giant":
        r *= 0.3
        r[7] = 2e-4
    elif case == "clusters":
        pos = np.repeat(rng.uniform(0.1 * L, 0.9 * L, (10, 3)), n // 10, axis=0) + rng.normal(0, 2e-5, (n, 3))
        r *= 0.2
    elif case == "zero and negative radii":
        r[::3] = 0.0
        r[1::5] = -1e-6
        pos[100:150] = pos[300:350]
    elif case == "outside the box":
        pos = pos * 1.5 - 0.2 * L
    elif case == "one cell":
        pos, r = pos[:120], r[:120] * 70
    elif case == "two cells":
        pos, r = pos[:300], r[:300] * 30
    elif case == "not finite":
        pos[5, 1] = np.nan
        pos[9, 0] = np.inf
    elif case == "far from the origin":
        pos = pos + np.array([1e3, -1e3, 50.0])
    elif case == "beyond FP32":
        pos, r = pos[:600] * 1e-39, r[:600] * 4e-39
    elif case == "partial last cell":
        r = np.clip(r, None, L / 2 / 24.5)
        r[0] = L / 2 / 24.5
    elif case == "list overflow":  # 244,650 pairs, the list holds 2 n + 65,536
        pos, r = pos[:700], np.full(700, 2 * L)
    elif case == "one droplet":
        pos, r = pos[:1], r[:1]
    return pos, r


@pytest.mark.parametrize("periodic", [True, False])
@pytest.mark.parametrize("case", ["uniform", "wide radii", "one giant", "clusters", "zero and negative radii",
                                  "outside the box", "one cell", "two cells", "not finite", "far from the origin",
                                  "beyond FP32", "partial last cell", "list overflow", "one droplet"])
def test_pair_set(case, periodic):
    from dem.collision_detector import SpatialHashCollisionDetector

    pos, r = _state(case)
    side = L * 1e-39 if case == "beyond FP32" else L
    det = SpatialHashCollisionDetector(len(r), L=side, boundary_mode="periodic" if periodic else "open")
    with np.errstate(all="ignore"):
        hit_ref, ref = O.hash_detect(pos, r, side, periodic, table_size=det._hash_table_size)
    hit, pairs = det.detect(pos, r)
    assert hit == hit_ref
    np.testing.assert_array_equal(pairs, ref)


@pytest.mark.parametrize("case", ["two cells", "list overflow"])
@pytest.mark.parametrize("cap", [0, 1, 57, 1000])
def test_short_buffer_holds_the_first_pairs(case, cap):
    import torch

    from dem import _native as N

    pos, r = _state(case)
    n = len(r)
    ctx = N.Context(n)
    table = 1 << (2 * n - 1).bit_length()
    _, ref = O.hash_detect(pos, r, L, True, table_size=table)
    soa = torch.as_tensor(np.ascontiguousarray(pos.T), device=ctx.device)
    pairs = torch.full((max(cap, 1), 2), -1, dtype=torch.int32, device=ctx.device)
    counts = torch.zeros(2, dtype=torch.int64, device=ctx.device)
    ctx.hash_detect(n, soa, torch.as_tensor(r, device=ctx.device), L, True, table, pairs, cap, counts)
    assert int(counts[0]) == len(ref) and ctx.device_errors() & N.DEVERR_PAIR_OVERFLOW
    np.testing.assert_array_equal(pairs.cpu().numpy()[:cap], ref[:cap])
