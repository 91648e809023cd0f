"""Multipoles formed in leaves and shifted up, and local expansions shifted
down: with two distant clusters accepted as one pair of cells, the truncated
field of one at the other does not depend on how far the clusters are split
below that pair, since a truncated multipole or local expansion shifts
exactly."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# the same FP64 sums grouped by other centres: at order 8 some 1e3 terms, each
# a few powers of offsets of the size of the cell
TOL = 1e-11
N = 420


@pytest.mark.parametrize("order", [1, 2, 3, 4, 5, 6, 7, 8])
@pytest.mark.parametrize("leaf", [1, 3, 32, 33, 64, 65, 128, 129, 300])
def test_field_of_a_cluster_does_not_depend_on_the_leaves(sim, order, leaf):
    rng = np.random.default_rng(100 * order + leaf)
    a = rng.random((N, 3)) * 0.2
    b = rng.random((N, 3)) * 0.2 + 0.8
    x, y, z = (np.concatenate([a[:, k], b[:, k]]) * 1e-3 for k in range(3))
    # the second cluster's own field is 1e-30 of the first one's
    q = np.concatenate([rng.random(N) + 0.5, np.full(N, 1e-30)]) * 1.6e-19
    # an opening of 3 takes the two clusters' depth-1 cells as one pair for every capacity
    f = np.array(sim.solve_fmm(x, y, z, q, order, 3.0, leaf_capacity=leaf))[:, N:]
    g = np.array(sim.solve_fmm(x, y, z, q, order, 3.0, leaf_capacity=N))[:, N:]
    assert sim.fmm_stats()["m2l_pairs"] == 2
    assert np.max(np.abs(g)) > 0.0
    assert np.max(np.abs(f - g)) <= TOL * np.max(np.abs(g))
