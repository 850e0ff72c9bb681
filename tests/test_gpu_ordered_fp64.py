"""The FP64 direct passes (csrc/direct_fp64.cu) at the edges of their tiles and row blocks, and on
operands outside the range of the branch-free square root and quotients: bit-identical to the oracle,
which adds the pair terms in the reference's order."""

from __future__ import annotations

import numpy as np
import pytest

import oracle as O
from gpu_util import consts

pytestmark = pytest.mark.gpu


def _check(pos, r, L, periodic):
    from dem.force_calculator import DirectDropletForceCalculator

    m, eta, _ = consts()
    fc = DirectDropletForceCalculator(num_particles=len(r), eta_oil=0.06, L=L,
                                      boundary_mode="periodic" if periodic else "open")
    F, V = fc.calculate_forces_and_convection(pos, r)
    F_ref = O.direct_forces(pos, r, m, L, periodic)
    np.testing.assert_array_equal(F, F_ref)
    np.testing.assert_array_equal(V, O.direct_convection(pos, F_ref, eta, L, periodic))


# tiles of 128 j's (4 and 8 rows) and 64 (16 rows); 4 rows to 1,776 droplets, 8 to 14,060 on 148 SMs
@pytest.mark.parametrize("periodic", [True, False])
@pytest.mark.parametrize("n", [1, 2, 5, 127, 128, 129, 1776, 1777, 2049, 14060, 14061])
def test_tile_and_row_edges(n, periodic):
    rng = np.random.default_rng(n)
    L = 3e-5 * n ** (1 / 3)
    _check(rng.uniform(0, L, (n, 3)), rng.uniform(1e-6, 8e-6, n), L, periodic)


@pytest.mark.parametrize("case", ["far below", "far above", "one far droplet", "zero radii", "on an axis", "coincident",
                                  "half box", "not finite"])
def test_operands_outside_the_fast_range(case):
    rng = np.random.default_rng(7)
    n, L = 300, 2e-4
    pos, r = rng.uniform(0, L, (n, 3)), rng.uniform(1e-6, 8e-6, n)
    periodic = case in ("far below", "half box", "on an axis")
    if case == "far below":  # r^2 < 2^-200
        pos, r, L = pos * 1e-38, r * 1e-38, L * 1e-38
    elif case == "far above":
        pos, r = pos * 1e40, r * 1e40
    elif case == "one far droplet":
        pos[40] = 1e35
    elif case == "zero radii":
        r[::7] = 0.0
    elif case == "on an axis":
        pos[:, 0] = 0.0
        pos[::3, 1] = 0.0
        pos[1, 2] = 1e-120
    elif case == "coincident":
        pos[11] = pos[12]
    elif case == "half box":  # separations of exactly L / 2
        L = 2.0**-12
        pos = rng.integers(0, 16, (n, 3)) * (L / 16) + np.arange(n)[:, None] * 2.0**-40
    elif case == "not finite":
        pos[5, 1] = np.inf
        pos[200, 0] = np.nan
    with np.errstate(all="ignore"):
        _check(pos, r, L, periodic)
