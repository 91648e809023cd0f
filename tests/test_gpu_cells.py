"""Pairs within a radius: the all-pairs kernels of small sets and the dense
grid of larger ones, at the sizes where one gives way to the other and on
clouds that strain the grid (one cell, flat, far outliers, dead, neutral and
non-finite particles), against the oracle."""
import numpy as np
import pytest

import oracle_lib as O

pytestmark = pytest.mark.gpu

E = 1.602176634e-19
TOL = 1e-12  # FP64 sums of at most a few hundred terms: n * 2^-53, with margin


def _cloud(n, seed, shape):
    rng = np.random.default_rng(seed)
    p = rng.normal(0.0, 1e-4, (3, n))
    if shape == "flat":
        p[2] = 0.0
    elif shape == "outlier":
        p[:, 0] = [0.5, -0.3, 0.9]
    elif shape == "duplicate":
        p[:, n // 2:] = p[:, : n - n // 2]
    return p[0], p[1], p[2], np.where(rng.random(n) < 0.5, E, -E)


@pytest.mark.parametrize("n", [1, 31, 33, 1024, 4096, 4097, 20011])
@pytest.mark.parametrize("shape", ["round", "flat", "outlier", "duplicate"])
def test_cutoff_forces(sim, n, shape):
    x, y, z, q = _cloud(n, n, shape)
    q[::7] = 0.0
    rc = 3e-4 if n < 5000 else 6e-6
    f = sim.solve_cutoff(x, y, z, q, rc)
    g = O.cutoff(x, y, z, q, rc)
    for a, b in zip(f, g):
        assert np.max(np.abs(a - b)) <= TOL * max(np.max(np.abs(b)), 1e-300)
    again = sim.solve_cutoff(x, y, z, q, rc)
    for a, b in zip(f, again):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("n", [4000, 5000])
def test_cutoff_leaves_out_non_finite(sim, n):
    x, y, z, q = _cloud(n, 5, "round")
    keep = np.ones(n, bool)
    keep[::11] = False
    xs = x.copy()
    xs[~keep] = np.nan
    xs[0] = np.inf
    f = sim.solve_cutoff(xs, y, z, q, 2e-5)
    g = O.cutoff(x[keep], y[keep], z[keep], q[keep], 2e-5)
    for a, b in zip(f, g):
        assert np.all(a[~keep] == 0.0)
        assert np.max(np.abs(a[keep] - b)) <= TOL * np.max(np.abs(b))


@pytest.mark.parametrize("n", [3, 200, 1024, 1025, 4096, 4097, 30001])
@pytest.mark.parametrize("species", [(1, 3), (1, 0), (0, 4)])
def test_annihilation_sets(n, species):
    import amk
    rng = np.random.default_rng(n)
    x, y, z = rng.normal(0.0, 1e-4, (3, n))
    sp = np.where(rng.random(n) < 0.5, species[0], species[1]).astype(np.uint8)
    radius = 1.2e-4 * n ** (-1.0 / 3.0)
    p = amk.make_params(seed=7, populations={"positron": n}, cutoff_radius=1e-5, annihilation_enabled=1,
                        contact_radius=radius, annihilation_probability=0.6, coulomb_forces_enabled=0)
    with amk.Simulation(p) as s:
        v = np.zeros(n)
        s.set_particles(x, y, z, v, v, v, sp)
        dead = np.ones(n, np.uint8)
        dead[::13] = 0
        amk.check(amk.lib().amk_set_alive(s.handle, dead.ctypes.data_as(amk._u8p)))
        marked = s.annihilate()
        alive = s.get_particles()["alive"]
        assert s.annihilate() >= 0  # a second search on the words the first left
    m, q = O.species_props(sp)
    ref = dict(x=x, y=y, z=z, vx=v, vy=v, vz=v, q=q, m=m, species=sp, alive=dead.copy())
    expect = O.annihilation(ref, radius, 0.6, 7, 1)
    assert marked == expect
    assert np.array_equal(alive, ref["alive"])
