"""The periodic-image correction of the direct passes at the edges of their
groups: the FP64 pass (csrc/direct_fp64.cu; four rows of a pair's j share the
table's reads) against the oracle, bit for bit, also where tiles take their terms
the general way (tiny coordinates); the FP32 pass (csrc/corr.cu; 32 targets per
CTA, runs of 32 terms, chunks of 64, tiles of 256) against the FP64 one.

FP32 tolerance, per droplet, of S = sum over j of max|G| (|Fx| + |Fy| + |Fz|) common:
the FP32 separation is 2.4e-7 L off at most, and the grid coordinate 4e-7 m cells
(m cells per axis) with the rounding of its two factors; a step between
neighbouring nodes is at most 2 max|G|, over three axes 2.4e-6 m.  Coefficients
(up to 8 max|G|), evaluation, factors and the sum of a run add 8e-6."""

from __future__ import annotations

import numpy as np
import pytest

import oracle as O
from gpu_util import ETA_OIL, consts, lognormal_state
from test_gpu_correction import _direct, _self_coeff

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


@pytest.mark.parametrize("tiny", [False, True])
@pytest.mark.parametrize("periodic", [True, False])
@pytest.mark.parametrize("n", [1, 2, 3, 5, 63, 64, 65, 129, 1776, 1777])
def test_fp64_pass_sizes(golden, n, periodic, tiny):
    g = golden("corr_direct_comsol_periodic_n64.npz" if periodic else "corr_direct_synth_open_n40.npz")
    pos, r, L = lognormal_state(n, seed=n, periodic=periodic)
    if tiny:
        pos[n // 2, n % 3] = 1e-95
    F = np.random.default_rng(n).normal(size=(n, 3))
    corr = O.Correction(g["grid_u"], g["grid_v"], g["grid_w"], g["grid_min"], g["grid_dx"], g["Fz_comsol"],
                        g["L_comsol"], g["eta_comsol"], L, ETA_OIL, _self_coeff(g, L))
    fc = _direct(n, L, periodic, g)
    V = fc.calculate_convection(pos, r, F)
    np.testing.assert_array_equal(V, O.direct_convection_corr(pos, F, consts()[1], L, periodic, corr))
    assert fc._ctx.device_errors() == 0
