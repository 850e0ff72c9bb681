"""Collision search of dense boxes: where the pairs are listed (the workspace, the output buffer, nowhere), how rows
of every length are sorted, and what a pair buffer keeps whose end falls into a row or between two.  The oracle's
pair sets."""

from __future__ import annotations

import functools

import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu

BOXES = {  # n, radius / L, periodic: pairs (the list holds 2 n + 65,536 in the workspace, 4.2 times that in the output)
    "rows up to 899": (900, 2.0, False),  # 404,550: more than either list
    "rows up to 699": (700, 2.0, False),  # 244,650: the output's list, j alone in the rows
    "rows of 60": (3000, 0.13, True),  # ~110,000 in periodic cells that repeat: the output's list, pairs in the rows
    "rows of 13": (2500, 0.08, False),  # ~32,000: the workspace's list
}


@functools.lru_cache(maxsize=None)
def _box(name):
    n, f, periodic = BOXES[name]
    rng = np.random.default_rng(n)
    pos, r = rng.uniform(0, 1.0, (n, 3)), np.full(n, f)
    r[::3] *= 0.9
    hit, ref = O.hash_detect(pos, r, 1.0, periodic, table_size=8192)
    return pos, r, periodic, ref


@pytest.mark.parametrize("where", ["empty", "first row", "workspace list", "past it", "row end", "pairs in rows", "past them",
                                   "output list", "past that", "all but one", "all", "all and more"])
@pytest.mark.parametrize("box", list(BOXES))
def test_pairs_and_buffer(box, where):
    import torch

    from dem import _native as N

    pos, r, periodic, ref = _box(box)
    n, total, half = len(r), len(ref), 2 * len(r) + 65536
    ends = np.flatnonzero(np.diff(ref[:, 0])) + 1
    cap = {"empty": 0, "first row": int(ends[0]) // 2, "workspace list": half, "past it": half + 1,
           "row end": int(ends[len(ends) // 2]), "pairs in rows": 2 * half, "past them": 2 * half + 1,
           "output list": 4 * half, "past that": 4 * half + 1, "all but one": total - 1, "all": total,
           "all and more": total + 1000}[where]
    ctx = N.Context(n)
    soa = torch.as_tensor(np.ascontiguousarray(pos.T), device=ctx.device)
    pairs = torch.full((cap + 1, 2), -7, dtype=torch.int32, device=ctx.device)
    counts = torch.zeros(2, dtype=torch.int64, device=ctx.device)
    ctx.hash_detect(n, soa, torch.as_tensor(r, device=ctx.device), 1.0, periodic, 8192, pairs, cap, counts)
    assert int(counts[0]) == total
    assert bool(ctx.device_errors() & N.DEVERR_PAIR_OVERFLOW) == (total > cap)
    got = pairs.cpu().numpy()
    np.testing.assert_array_equal(got[: min(cap, total)], ref[:cap])
    assert (got[cap] == -7).all()


@pytest.mark.parametrize("n,phi", [(20000, 0.6), (20000, 2.0), (40000, 0.3), (40000, 3.0)])
@pytest.mark.parametrize("periodic", [True, False])
def test_volume_fractions(n, phi, periodic):
    from dem.collision_detector import SpatialHashCollisionDetector

    rng = np.random.default_rng(n)
    r = np.full(n, 5e-6) * (1 + 0.3 * rng.random(n))
    L = float((4 / 3 * np.pi * (r**3).sum() / phi) ** (1 / 3))
    pos = rng.uniform(0, L, (n, 3))
    det = SpatialHashCollisionDetector(n, L=L, boundary_mode="periodic" if periodic else "open")
    _, ref = O.hash_detect(pos, r, L, periodic, table_size=det._hash_table_size)
    _, pairs = det.detect(pos, r)
    np.testing.assert_array_equal(pairs, ref)
