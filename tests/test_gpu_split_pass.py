"""The mixed passes' split schedule (csrc/direct_mixed.cu) at the edges of its runs (64 j's), of its warps'
near-pair queue (32 pairs a round) and of the sizes that choose its rows per thread and packing kernel:
against the FP64 passes, with the mixed precision's own bounds, and the same bits in two calls."""

from __future__ import annotations

import numpy as np
import pytest

from gpu_util import rel_norm

pytestmark = pytest.mark.gpu


def _both(pos, r, L, periodic, schedule="split"):
    from dem.force_calculator import DirectDropletForceCalculator

    out = []
    for precision in ("fp64", "mixed"):
        fc = DirectDropletForceCalculator(num_particles=len(r), eta_oil=0.06, L=L, precision=precision,
                                          boundary_mode="periodic" if periodic else "open")
        fc.set_tuning(schedule=schedule)
        out.append(fc.calculate_forces_and_convection(pos, r))
        again = fc.calculate_forces_and_convection(pos, r)
        assert all(np.array_equal(a, b) for a, b in zip(out[-1], again))
        assert fc._ctx.device_errors() == 0
    (F, V), (Fm, Vm) = out
    return rel_norm(Fm, F), rel_norm(Vm, V)


@pytest.mark.parametrize("periodic", [True, False])
@pytest.mark.parametrize("n", [2, 31, 63, 64, 65, 127, 129, 2000, 4033, 12288, 12289, 16384, 16385])
def test_run_and_plan_edges(n, periodic):
    rng = np.random.default_rng(n)
    L = 3.5e-5 * n ** (1 / 3)
    ef, ev = _both(rng.uniform(0, L, (n, 3)), rng.uniform(2e-6, 8e-6, n), L, periodic)
    assert ef <= 1e-6 and ev <= 2e-6  # the bounds of the mixed passes' own tests


def test_dense_clusters_fill_the_queue():
    """Every pair of a warp's run near: 64 entries per lane, 64 rounds."""
    rng = np.random.default_rng(3)
    n, L = 640, 1e-3
    centres = np.repeat(rng.uniform(0.2 * L, 0.8 * L, (5, 3)), 128, axis=0)
    pos = centres + rng.uniform(-1e-5, 1e-5, (n, 3))
    ef, ev = _both(pos, np.full(n, 2e-6), L, True)
    assert ef <= 1e-6 and ev <= 2e-6
