"""The symmetric mixed passes (csrc/direct_mixed_sym.cu) where a box's last block is nearly all padding, one
sub-tile (32 entries) or run (64) from it, or whole, with the diagonal items split in two: against the FP64
passes, with the mixed precision's own bounds, and the same bits in two calls."""

from __future__ import annotations

import numpy as np
import pytest

from gpu_util import rel_norm

pytestmark = pytest.mark.gpu


def _passes(pos, r, L, periodic, precision, **tuning):
    from dem.force_calculator import DirectDropletForceCalculator

    fc = DirectDropletForceCalculator(num_particles=len(r), eta_oil=0.06, L=L, precision=precision,
                                      boundary_mode="periodic" if periodic else "open")
    if tuning:
        fc.set_tuning(**tuning)
    out = fc.calculate_forces_and_convection(pos, r)
    assert all(np.array_equal(a, b) for a, b in zip(out, fc.calculate_forces_and_convection(pos, r)))
    assert fc._ctx.device_errors() == 0
    return out


def _box(n):
    rng = np.random.default_rng(n)
    L = 3.5e-5 * n ** (1 / 3)
    return rng.uniform(0, L, (n, 3)), rng.uniform(2e-6, 8e-6, n), L


@pytest.mark.parametrize("periodic", [True, False])
@pytest.mark.parametrize("rows", [2, 4])
@pytest.mark.parametrize("n", [2, 32, 33, 64, 65, 255, 257, 511, 513, 544, 545, 577, 1023, 4097, 8193])
def test_last_block(n, rows, periodic):
    pos, r, L = _box(n)
    F, V = _passes(pos, r, L, periodic, "fp64")
    Fm, Vm = _passes(pos, r, L, periodic, "mixed", schedule="symmetric", i_per_thread=rows)
    assert rel_norm(Fm, F) <= 1e-6 and rel_norm(Vm, V) <= 2e-6  # the bounds of the mixed passes' own tests
