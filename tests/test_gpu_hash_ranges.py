"""Collision search with radii and positions at the ends of FP64's range: infinite radii, radii above FP32's
largest and below its smallest number, radii whose squares underflow, positions at infinity among droplets
that touch (the oracle's pair sets); and more pairs than 32 bits count."""

from __future__ import annotations

import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


def _state(case, n=600):
    rng = np.random.default_rng(len(case))
    L = 1.0
    pos, r = rng.uniform(0, L, (n, 3)), rng.uniform(0.02, 0.05, n)
    if case == "one infinite radius":
        r[7] = np.inf
    elif case == "infinite radii":
        r[::2] = np.inf
    elif case == "one radius of 1e39":
        r[7] = 1e39
    elif case == "radii of 1e39":
        r *= 1e40
        r[3] = 0.02
    elif case == "radii near the largest number":  # the sum of two overflows
        r = r / 0.05 * 1.7e308
    elif case == "positions at infinity":
        pos[5::17, 0] = np.inf
        pos[6::23, 2] = -np.inf
        pos[8::41] = np.inf
    elif case == "scaled by 1e-45":
        L, pos, r = L * 1e-45, pos * 1e-45, r * 1e-45
    elif case == "scaled by 1e-100":
        L, pos, r = L * 1e-100, pos * 1e-100, r * 1e-100
    elif case == "scaled by 1e-160":  # squares of separations and radii sums are subnormal or zero
        L, pos, r = L * 1e-160, pos * 1e-160, r * 1e-160
    elif case == "scaled by 1e-306":
        L, pos, r = L * 1e-306, pos * 1e-306, r * 1e-306
    elif case == "radii of 1e-200 in a unit box":
        pos[300:] = pos[:300] + 1e-170
        r *= 1e-198
    elif case == "scaled by 1e100":
        L, pos, r = L * 1e100, pos * 1e100, r * 1e100
    return pos, r, L


@pytest.mark.parametrize("periodic", [True, False])
@pytest.mark.parametrize("case", ["one infinite radius", "infinite radii", "one radius of 1e39", "radii of 1e39",
                                  "radii near the largest number", "positions at infinity", "scaled by 1e-45", "scaled by 1e-100", "scaled by 1e-160",
                                  "scaled by 1e-306", "radii of 1e-200 in a unit box", "scaled by 1e100"])
def test_pair_set(case, periodic):
    from dem.collision_detector import SpatialHashCollisionDetector

    pos, r, L = _state(case)
    det = SpatialHashCollisionDetector(len(r), L=L, boundary_mode="periodic" if periodic else "open")
    with np.errstate(all="ignore"):
        hit_ref, ref = O.hash_detect(pos, r, L, periodic, table_size=det._hash_table_size)
    hit, pairs = det.detect(pos, r)
    assert hit == hit_ref
    np.testing.assert_array_equal(pairs, ref)


def test_more_than_2_32_pairs():
    """92,683 coincident droplets have 2^32 + 55,607 pairs: a count modulo 2^32 would fit the list."""
    import torch

    from dem import _native as N

    n, cap = 92683, 16
    total = n * (n - 1) // 2
    ctx = N.Context(n)
    assert 0 < total - 2**32 < 2 * n + 65536
    soa = torch.full((3, n), 0.5, dtype=torch.float64, device=ctx.device)
    r = torch.full((n,), 0.01, dtype=torch.float64, device=ctx.device)
    pairs = torch.full((cap, 2), -1, dtype=torch.int32, device=ctx.device)
    counts = torch.zeros(2, dtype=torch.int64, device=ctx.device)
    ctx.hash_detect(n, soa, r, 1.0, True, 1 << 18, pairs, cap, counts)
    assert int(counts[0]) == total and ctx.device_errors() & N.DEVERR_PAIR_OVERFLOW
    np.testing.assert_array_equal(pairs.cpu().numpy(), [[0, j] for j in range(1, cap + 1)])
