"""Training tiles of the correction's network: gradients at the edges of the
8-, 16- and 32-sample tiles and of one and several tiles per CTA, against the
FP64 restatement (oracle/mlp_oracle.py)."""
import numpy as np
import pytest

import mlp_oracle as MO

pytestmark = pytest.mark.gpu

# a gradient element is an FP32 sum of n products (forward error of a few
# 128-long FMA chains each): 128 * 2^-24 * 4 layers = 3e-5 of the largest
# element bounds the products' error, the sums' own error is below it
TOL = 1e-4


@pytest.mark.parametrize("n", [1, 7, 8, 9, 8 * 148, 8 * 148 + 1, 16 * 148, 16 * 148 + 3, 32 * 148, 32 * 148 + 1, 9999])
def test_gradients_at_tile_edges(sim, n):
    p = MO.init_params(n % 91)
    sim.set_mlp_params(p)
    rng = np.random.default_rng(n)
    x = rng.normal(0, 1, (n, MO.IN)).astype(np.float32)
    t = rng.normal(0, 1, (n, 3)).astype(np.float32)
    loss, g, y = sim.mlp_gradients(x, t)
    rloss, rg = MO.gradients(p, x, t)
    assert abs(loss - rloss) <= 1e-5 * abs(rloss)
    assert np.max(np.abs(y - MO.forward(p, x))) < TOL * np.max(np.abs(y))
    off = 0
    for name, shape in MO.SHAPES:
        k = int(np.prod(shape))
        a, b = g[off:off + k], rg[off:off + k]
        assert np.max(np.abs(a - b)) <= TOL * (np.max(np.abs(b)) + 1e-30), name
        off += k
    again = sim.mlp_gradients(x, t)[1]
    assert np.array_equal(g, again)  # the tiles' parts are added in a fixed order
