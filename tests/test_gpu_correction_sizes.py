"""The FP32 pass of the periodic-image correction (csrc/corr.cu) at the edges of
its target groups (32 per CTA), runs (32 terms), chunks (64) and tiles (256),
against the FP64 correction, which is bit-identical to the reference's.

Tolerance, per droplet, of S = sum over j of max|G| (|Fx| + |Fy| + |Fz|) common:
the FP32 separation is 2.4e-7 L off at most, and the grid coordinate 4e-7 m cells
(m cells per axis) with the rounding of its two factors; a step between
neighbouring nodes is at most 2 max|G|, over three axes 2.4e-6 m.  Coefficients
(up to 8 max|G|), evaluation, factors and the sum of a run add 8e-6."""

from __future__ import annotations

import numpy as np
import pytest

from gpu_util import lognormal_state
from test_gpu_correction import _direct

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("periodic", [True, False])
@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 63, 64, 65, 255, 256, 257, 1000, 3001])
def test_fp32_pass_sizes(golden, n, periodic):
    g = golden("corr_direct_comsol_periodic_n64.npz" if periodic else "corr_direct_synth_open_n40.npz")
    pos, r, L = lognormal_state(n, seed=n, periodic=periodic)
    F = np.random.default_rng(n).normal(size=(n, 3))
    corr = {}
    for precision in ("mixed", "fp64"):
        fc = _direct(n, L, periodic, g, precision=precision)
        with_corr = fc.calculate_convection(pos, r, F)
        common = fc._corr.info()["common"]
        fc._corr = None
        corr[precision] = with_corr - fc.calculate_convection(pos, r, F)
        assert fc._ctx.device_errors() == 0
    big = max(np.abs(g[k]).max() for k in ("grid_u", "grid_v", "grid_w"))
    S = abs(common) * big * np.abs(F).sum()
    m = len(g["grid_u"]) - 1
    assert np.abs(corr["mixed"] - corr["fp64"]).max() <= (2.4e-6 * m + 8e-6) * S
