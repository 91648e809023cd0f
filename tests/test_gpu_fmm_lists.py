"""Interaction lists grouped by target: groups of every size the sorts tell
apart (a warp's registers, a block's shared memory, in place) give the exact
sum at theta = 0, where every leaf's near-field list holds every leaf, and the
same forces on every run."""
import numpy as np
import pytest

import oracle_lib as O
from conftest import gaussian_cloud, rel_errors

pytestmark = pytest.mark.gpu

# FP64 sums of n terms in another order than the oracle's, relative to a force
# that mixed charges may cancel by a few orders: the FMM fixtures' 1e-9
TOL = 1e-9


@pytest.mark.parametrize("n,leaf", [(40, 32), (60, 2), (600, 8), (1500, 8), (3000, 8), (6000, 8), (9000, 4),
                                    (16700, 1)])
def test_theta_zero_lists(sim, n, leaf):
    x, y, z, q = gaussian_cloud(n, n)
    f = sim.solve_fmm(x, y, z, q, 2, 0.0, leaf_capacity=leaf)
    rel, _ = rel_errors(f, O.allpairs(x, y, z, q))
    assert np.max(rel) < TOL
    again = sim.solve_fmm(x, y, z, q, 2, 0.0, leaf_capacity=leaf)
    for a, b in zip(f, again):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("order", [1, 2, 3, 4, 5, 6, 7, 8])
@pytest.mark.parametrize("n,theta,leaf", [(700, 0.5, 8), (5000, 0.3, 4), (20000, 0.6, 64)])
def test_harmonic_basis_products(sim, monkeypatch, order, n, theta, leaf):
    # class products against the per-pair path (a class reach of 0 sends every
    # pair there), whose derivatives come from the actual centres; both sum
    # the same FP64 terms, so they differ by rounding: 1e-12 of the force scale
    x, y, z, q = gaussian_cloud(n, order, mixed=False)
    f = sim.solve_fmm(x, y, z, q, order, theta, leaf_capacity=leaf)
    st = sim.fmm_stats()
    assert st["m2l_class_pairs"] > 0
    monkeypatch.setenv("AMK_FMM_M2L_REACH", "0")
    g = sim.solve_fmm(x, y, z, q, order, theta, leaf_capacity=leaf)
    assert sim.fmm_stats()["m2l_class_pairs"] == 0
    scale = max(np.max(np.abs(b)) for b in g)
    for a, b in zip(f, g):
        assert np.max(np.abs(a - b)) <= 1e-12 * scale
