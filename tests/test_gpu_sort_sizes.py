"""The Morton sort (csrc/bh.cu) at the edges of its cluster kernel's rounds (8,192 pairs each, up to 65,536)
and of the tiled passes past it: the symmetric passes, which take their blocks from it, against the FP64
passes with the mixed precision's own bounds, and the same bits as a second call."""

from __future__ import annotations

import numpy as np
import pytest

from gpu_util import rel_norm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("periodic", [True, False])
@pytest.mark.parametrize("n", [1, 2, 33, 8191, 8192, 8193, 16385, 65535, 65536, 65537])
def test_symmetric_passes(n, periodic):
    from dem.force_calculator import DirectDropletForceCalculator

    rng = np.random.default_rng(n)
    L = 3.5e-5 * n ** (1 / 3)
    pos, r = rng.uniform(0, L, (n, 3)), rng.uniform(2e-6, 8e-6, n)
    pos[n // 2:] = pos[n // 2:][:, [0, 0, 0]]  # half the droplets on a diagonal: equal digits in a row
    out = []
    for precision in ("fp64", "mixed"):
        fc = DirectDropletForceCalculator(num_particles=n, eta_oil=0.06, L=L, precision=precision,
                                          boundary_mode="periodic" if periodic else "open")
        fc.set_tuning(schedule="symmetric")
        out.append(fc.calculate_forces_and_convection(pos, r))
        if precision == "mixed":
            again = fc.calculate_forces_and_convection(pos, r)
            assert all(np.array_equal(a, b) for a, b in zip(out[-1], again))
    (F, V), (Fm, Vm) = out
    if n > 1:
        assert rel_norm(Fm, F) <= 1e-6 and rel_norm(Vm, V) <= 2e-6  # the bounds of the mixed passes' own tests
