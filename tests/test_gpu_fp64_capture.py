"""The FP64 passes under stream capture as the first calls of their context (csrc/direct_fp64.cu raises a kernel's
shared-memory limit in the call that first takes it): the replay leaves the bits of an eager call."""

from __future__ import annotations

import numpy as np
import pytest

from gpu_util import consts

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("periodic", [True, False])
@pytest.mark.parametrize("n", [100, 1777, 14061])  # 4, 8 and 16 rows per CTA
def test_first_calls_captured(n, periodic):
    import torch

    from dem import _native as N

    m, eta, _ = consts()
    L = 3e-5 * n ** (1 / 3)
    g = torch.Generator("cuda").manual_seed(n)
    pos = L * torch.rand((3, n), device="cuda", dtype=torch.float64, generator=g)
    r = 1e-6 + 6e-6 * torch.rand(n, device="cuda", dtype=torch.float64, generator=g)
    out = []
    for captured in (True, False):
        ctx = N.Context(n)
        F, V = torch.empty_like(pos), torch.empty_like(pos)

        def passes():
            ctx.direct_forces(n, pos, r, m, L, periodic, N.PREC_FP64, F)
            ctx.direct_convection(n, pos, r, F, eta, L, periodic, N.PREC_FP64, V)

        if captured:
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph):
                passes()
            graph.replay()
        else:
            passes()
        assert ctx.device_errors() == 0
        out.append((F.cpu().numpy(), V.cpu().numpy()))
    for a, b in zip(*out):
        assert np.abs(a).sum() > 0
        np.testing.assert_array_equal(a, b)
