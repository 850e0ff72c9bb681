"""The queue-fed Morton-tree walks (csrc/bh.cu, from 131,072 targets): sampled rows of force and velocity against the
oracle's direct sums, at theta = 0 (every pair) and at theta = 0.5 within the bounds of test_gpu_morton_tree.py.

At theta = 0 a pair's force errs with its separation: FP32 coordinates from the box centre are off by 2^-26 L each, a
separation by up to sqrt(3) 2^-25 L, and |F| ~ |d|^-4 with |d| >= r_i + r_j."""

from __future__ import annotations

import numpy as np
import pytest

import oracle as O
from gpu_util import ETA_OIL, consts, lognormal_state, rel_norm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("periodic", [True, False])
@pytest.mark.parametrize("n", [131072, 131073])
def test_sampled_rows(n, periodic):
    from dem.octree import MortonTreeForceCalculator, TreeDropletForceCalculator

    pos, r, L = lognormal_state(n, seed=n, periodic=periodic)
    # a shuffled sample at the front, so that the rows come from all over the box
    order = np.random.default_rng(n).permutation(n)
    pos, r = np.ascontiguousarray(pos[order]), np.ascontiguousarray(r[order])
    rows = (0, 512)
    m, eta, _ = consts()
    kw = dict(num_particles=n, mpl=16, eta_oil=ETA_OIL, L=L, periodic=periodic)
    touching = 4 * 3**0.5 * 2.0**-25 * L / (2 * r.min())  # 1.7e-4 and 1.9e-4
    for theta, bound in ((0.0, touching), (0.5, 1.5e-3)):
        tc = MortonTreeForceCalculator(theta=theta, window_level=4, **kw)
        F, V = tc.calculate_forces_and_convection(pos, r)
        F_ref = O.direct_forces(pos, r, m, L, periodic, rows=rows)[: rows[1]]
        V_ref = O.direct_convection(pos, F, eta, L, periodic, rows=rows)[: rows[1]]  # the walk's own forces in
        assert rel_norm(F[: rows[1]], F_ref) <= bound
        err = rel_norm(V[: rows[1]], V_ref)
        if theta == 0.0:
            assert err <= 2e-5
            assert tc.stats()["node_terms"] == 0 and tc.stats()["leaf_pairs"] == n * n
        else:
            parity = TreeDropletForceCalculator(theta=theta, **kw)
            Fp, Vp = parity.calculate_forces_and_convection(pos, r)
            Vp_ref = O.direct_convection(pos, Fp, eta, L, periodic, rows=rows)[: rows[1]]
            assert err <= 1.1 * rel_norm(Vp[: rows[1]], Vp_ref)
        assert tc._ctx.device_errors() == 0
