"""The parity tree's walk records (csrc/tree.cu) where whole subtrees are passed over: droplets of radius
zero (R^3 sums below the reference's threshold), zero forces (its other threshold), every droplet in one
octant, coincident droplets in one leaf, one droplet, rebuilding on the same tree.  Bit-identical to the oracle."""

from __future__ import annotations

import numpy as np
import pytest

import oracle as O
from gpu_util import consts

pytestmark = pytest.mark.gpu


def _state(case, n, L):
    rng = np.random.default_rng(5)
    pos, r = rng.uniform(0, L, (n, 3)), rng.uniform(2e-6, 6e-6, n)
    F = rng.normal(size=(n, 3)) * 1e-12
    if case == "zero radii":
        r[pos[:, 0] < 0.6 * L] = 0.0
    elif case == "all zero radii":
        r[:] = 0.0
    elif case == "zero forces":
        F[pos[:, 1] < 0.7 * L] = 0.0
    elif case == "one octant":
        pos *= 0.01
    elif case == "coincident":
        pos[: n // 2] = pos[0]
    elif case == "one droplet":
        pos, r, F = pos[:1], r[:1], F[:1]
    return pos, r, F


@pytest.mark.parametrize("periodic", [True, False])
@pytest.mark.parametrize("mpl", [1, 3])
@pytest.mark.parametrize("case", ["zero radii", "all zero radii", "zero forces", "one octant", "coincident",
                                  "one droplet"])
def test_walks_bit_exact(case, mpl, periodic):
    from dem.octree import FlatOctree

    n, L = 1500, 4e-4
    m, eta, sf = consts()
    t = FlatOctree(theta=0.5, mpl=mpl, num_particles=n)
    pos, r, F_in = _state("", n, L)
    t.build(pos, r, L=L, periodic=periodic)  # a first tree, whose records must not be met again
    t.compute_forces_and_total_velocity(m, eta, sf)
    pos, r, F_in = _state(case, n, L)
    with np.errstate(all="ignore"):
        ref = O.Tree(n, 0.5, mpl)
        ref.build(pos, r, L, periodic)
        t.build(pos, r, L=L, periodic=periodic)
        F, V = t.compute_forces_and_total_velocity(m, eta, sf)
        F_ref, V_ref = ref.forces_and_total_velocity(m, eta, sf)
        np.testing.assert_array_equal(F, F_ref)
        np.testing.assert_array_equal(V, V_ref)
        t.build(pos, r, L=L, periodic=periodic)
        ref.build(pos, r, L, periodic)
        ref.propagate_forces(F_in)
        np.testing.assert_array_equal(t.compute_stokeslet(F_in, eta), ref.velocity(F_in, eta))
