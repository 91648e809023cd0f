"""Leaf depths at capacities around the window sizes of the sliding maximum
(256 particles, two windows and the part between above), against the ranges of
a recursive split on the host."""
import numpy as np
import pytest

from conftest import E
from test_gpu_sort import _expected_ranges

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 257, 3000, 20000])
@pytest.mark.parametrize("cap", [1, 2, 7, 8, 128, 254, 255, 256, 257, 511, 512, 1000, 2999, 3000, 100000])
def test_leaf_ranges(sim, n, cap):
    rng = np.random.default_rng(n + cap)
    x, y, z = rng.normal(0.0, [[1e-4], [1e-4], [3e-4]], (3, n))
    f, g = sim.bh_tree(x, y, z, np.full(n, E), leaf_capacity=cap)
    assert sorted(zip(g[:, 8].tolist(), g[:, 9].tolist())) == _expected_ranges(x, y, z, cap)


def test_coincident_particles(sim):
    # a cell at the key depth may hold more than the capacity
    n = 700
    x = np.repeat([1e-4, -1e-4], [n - 100, 100])
    f, g = sim.bh_tree(x, x, x, np.full(n, E), leaf_capacity=300)
    ends = sorted(zip(g[:, 8].tolist(), g[:, 9].tolist()))
    assert ends[0] == (0, 100) and ends[1] == (0, n)
    assert ends.count((100, n)) == 21
