"""A parity tree that the device has no memory for: the creation reports it, and the context's next calls do not."""

from __future__ import annotations

import numpy as np
import pytest

import oracle as O
from gpu_util import lognormal_state

pytestmark = pytest.mark.gpu


def test_failed_creation_leaves_no_error_behind():
    import torch

    from dem import _native as N

    n = 1000
    pos, r, L = lognormal_state(n, seed=5, volume_fraction=0.05)
    ctx = N.Context(n)
    soa = torch.as_tensor(np.ascontiguousarray(pos.T), device=ctx.device)
    pairs = torch.zeros((4 * n, 2), dtype=torch.int32, device=ctx.device)
    counts = torch.zeros(2, dtype=torch.int64, device=ctx.device)
    with pytest.raises(N.DemError, match="tree allocation"):
        N.Tree(ctx, n, 2**31 - 1)  # ~945 GB of nodes
    ctx.hash_detect(n, soa, torch.as_tensor(r, device=ctx.device), L, True, 2048, pairs, 4 * n, counts)
    _, ref = O.hash_detect(pos, r, L, True, table_size=2048)
    assert int(counts[0]) == len(ref)
    np.testing.assert_array_equal(pairs.cpu().numpy()[: len(ref)], ref)
