"""Partners on both sides of a cell in a long, thin cloud: with millions of
cells along one axis a cell coordinate's rounding may exceed the margin by which
a cell is wider than the radius."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

E = 1.602176634e-19
K = 8.9875517923e9
RC = 1e-6


# lowest x of the cloud and a pair just inside RC whose cells, RC (1 + 1e-9)
# wide from there, are two apart by the FP64 evaluation of (x - lowest) / width
@pytest.mark.parametrize("low,a,b", [
    (-0.0008645139872939852, 15.999844502013415, 15.999845502013414),
    (-0.0009301820814270931, 15.999524833919029, 15.999525833919028),
    (-0.0009535586353559682, 15.999755457365353, 15.999756457365352),
])
def test_pair_near_the_radius_in_a_thin_cloud(sim, low, a, b):
    inv = 1.0 / (RC * (1.0 + 1e-9))
    assert 0.0 < b - a < RC and np.floor((b - low) * inv) - np.floor((a - low) * inv) >= 2.0
    n = 1 << 22
    x = np.linspace(low, 15.9, n)  # 3.8 radii apart
    x[0], x[1] = low, 16.0  # the pair is inside the cloud
    x[-2:] = a, b
    o = np.zeros(n)
    fx, fy, fz = sim.solve_cutoff(x, o, o, np.full(n, E), RC)
    f = K * E * E / (b - a) ** 2
    assert abs(fx[-1] - f) <= 1e-12 * f and abs(fx[-2] + f) <= 1e-12 * f
    assert not np.any(fx[:-2]) and not np.any(fy) and not np.any(fz)
