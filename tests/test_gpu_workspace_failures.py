"""Workspaces whose growth fails: the call reports an error, and the context goes on with smaller sizes instead of
using memory that it no longer holds."""

from __future__ import annotations

import numpy as np
import pytest

import oracle as O
from gpu_util import lognormal_state

pytestmark = pytest.mark.gpu


@pytest.fixture
def nearly_full():
    """Device memory with at most 700 MB free."""
    import torch

    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    ballast = torch.empty(free - (700 << 20), dtype=torch.uint8, device="cuda")
    yield
    del ballast
    torch.cuda.empty_cache()


def test_reserve():
    import torch

    from dem import _native as N

    pos, r, L = lognormal_state(1000, seed=3, volume_fraction=0.05)
    pos += np.random.default_rng(0).normal(0, 3e-6, pos.shape)
    pos %= L
    ctx = N.Context(1000)
    soa = torch.as_tensor(np.ascontiguousarray(pos.T), device=ctx.device)
    rr = torch.as_tensor(r, device=ctx.device)
    pairs = torch.zeros((4000, 2), dtype=torch.int32, device=ctx.device)
    counts = torch.zeros(2, dtype=torch.int64, device=ctx.device)
    with pytest.raises(N.DemError):
        ctx.reserve(2**31 - 1)  # more than the device has
    assert ctx.capacity == 0
    with pytest.raises(ValueError, match="capacity"):
        ctx.hash_detect(1000, soa, rr, L, True, 2048, pairs, 4000, counts)
    ctx.reserve(1000)
    ctx.hash_detect(1000, soa, rr, L, True, 2048, pairs, 4000, counts)
    _, ref = O.hash_detect(pos, r, L, True, table_size=2048)
    assert len(ref) > 10
    np.testing.assert_array_equal(pairs.cpu().numpy()[: int(counts[0])], ref)


def test_partial_sums(nearly_full):
    import torch

    from dem import _native as N
    from dem.force_calculator import DirectDropletForceCalculator

    n = 65536
    g = torch.Generator("cuda").manual_seed(1)
    pos = 2e-3 * torch.rand((n, 3), dtype=torch.float64, device="cuda", generator=g)
    r = torch.full((n,), 5e-6, dtype=torch.float64, device="cuda")
    calc = DirectDropletForceCalculator(n, L=2e-3, precision="mixed")
    calc.set_tuning(schedule=N.SCHED_SPLIT, j_splits=8)
    first = [t.clone() for t in calc.calculate_forces_and_convection(pos, r)]
    calc.set_tuning(schedule=N.SCHED_SPLIT, j_splits=1024)  # 1.6 GB of partial sums
    with pytest.raises(N.DemError):
        calc.calculate_forces_and_convection(pos, r)
    calc.set_tuning(schedule=N.SCHED_SPLIT, j_splits=8)
    for a, b in zip(calc.calculate_forces_and_convection(pos, r), first):
        assert torch.equal(a, b)


def test_vjp_records():
    """Records of 1.1 GB: with room for half of them the same bits, from more and smaller launches."""
    import torch

    from dem import _native as N

    n, L = 65536, 2e-3
    g = torch.Generator("cuda").manual_seed(2)
    kw = dict(dtype=torch.float64, device="cuda", generator=g)
    pos, F, lam = L * torch.rand((3, n), **kw), torch.randn((3, n), **kw), torch.randn((3, n), **kw)
    r = 5e-6 * (0.5 + torch.rand(n, **kw))

    def vjp():
        out = [torch.zeros((3, n), dtype=torch.float64, device="cuda") for _ in range(2)] + [torch.zeros_like(r)]
        before = N.launch_count()
        N.Context(n).direct_vjp(n, pos, r, F, lam, 1e-9, 0.7, 1.3, L, True, *out)
        return out, N.launch_count() - before

    roomy, launches = vjp()
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    ballast = torch.empty(free - (700 << 20), dtype=torch.uint8, device="cuda")
    tight, more = vjp()
    del ballast
    torch.cuda.empty_cache()
    assert more > launches
    for a, b in zip(tight, roomy):
        assert torch.isfinite(a).all() and torch.equal(a, b)
