"""Cells of clouds that fill little of their bounding box, where the cell list
hashes them: cutoff forces, energies and annihilation against the oracle on both
sides of the rule (dense cells up to two radii wide), and the cost of one
particle far from the others."""
import time

import numpy as np
import pytest

import amk
import oracle_lib as O

pytestmark = pytest.mark.gpu

E = 1.602176634e-19
TOL = 1e-12  # FP64 sums of at most a few hundred terms: n * 2^-53, with margin


def _cloud(n, shape, seed):
    rng = np.random.default_rng(seed)
    p = rng.normal(0.0, 1e-4, (3, n))
    if shape == "far":       # one particle at a trap wall, one beyond it
        p[:, 5], p[:, 77] = [0.01, -0.008, 0.02], [-1.0, 3.0, 0.5]
    elif shape == "halo":    # a dense core in a thin halo
        p *= np.where(rng.random(n) < 0.1, 100.0, 0.3)
    elif shape == "clusters":
        p += 0.05 * rng.integers(0, 3, n)
    elif shape == "line":    # along one axis
        p[1:] = 0.0
        p[0] *= 50.0
    elif shape == "offset":  # far from the origin: few bits left inside the cloud
        p += 4.0
    return p[0], p[1], p[2]


def _radius(x, y, z, near):
    """A radius with about `near` partners inside it for a typical particle."""
    rng = np.random.default_rng(0)
    k = rng.integers(0, len(x), 64)
    d = np.sqrt((x[k, None] - x) ** 2 + (y[k, None] - y) ** 2 + (z[k, None] - z) ** 2)
    m = max(1, int(np.ceil(near)))
    return float(np.median(np.sort(d, axis=1)[:, m])) * (near / m) ** (1.0 / 3.0)


@pytest.mark.parametrize("n", [4097, 12011])
@pytest.mark.parametrize("shape", ["ball", "far", "halo", "clusters", "line", "offset"])
@pytest.mark.parametrize("near", [0.05, 1.0, 20.0])
def test_forces_energy_and_contacts(n, shape, near):
    x, y, z = _cloud(n, shape, n)
    r = _radius(x, y, z, near)
    sp = np.where(np.random.default_rng(1).random(n) < 0.5, 1, 3).astype(np.uint8)
    m, q = O.species_props(sp)
    p = amk.make_params(seed=7, populations={"positron": n}, coulomb_method="standard", cutoff_radius=r,
                        energy_method="standard", annihilation_enabled=1, contact_radius=r,
                        annihilation_probability=0.6)
    v = np.zeros(n)
    with amk.Simulation(p) as s:
        s.set_particles(x, y, z, v, v, v, sp)
        s.coulomb_standard(r)
        f = s.get_forces()
        s.coulomb_standard(r)
        again = s.get_forces()
        pot = s.energy(time_centre=False)["coulomb_potential"]
        marked = s.annihilate()
        alive = s.get_particles()["alive"]
    g = O.cutoff(x, y, z, q, r)
    scale = max(np.max(np.abs(b)) for b in g)
    for a, b, c in zip(f, g, again):
        assert np.max(np.abs(a - b)) <= TOL * scale
        assert np.array_equal(a, c)
    ref = dict(x=x, y=y, z=z, vx=v, vy=v, vz=v, q=q, m=m, species=sp, alive=np.ones(n, np.uint8))
    coul = O.energy_standard(ref, p.trap_voltage, p.z0, p.rho0, r)["coulomb_potential"]
    size = 0.5 * 8.9875517923e9 * E * E * n / r  # of the sum's terms
    assert abs(pot - coul) <= 1e-12 * max(size, abs(coul))
    assert marked == O.annihilation(ref, r, 0.6, 7, 1)
    assert np.array_equal(alive, ref["alive"])


def test_one_far_particle_costs_little(sim):
    # 100 times and more with cells as wide as the box asks for
    n = 200003
    rng = np.random.default_rng(2)
    x, y, z = rng.normal(0.0, 1e-4, (3, n))
    q = np.where(rng.random(n) < 0.5, E, -E)

    def seconds(far):
        x[0] = y[0] = z[0] = far
        t = []
        for _ in range(6):
            t0 = time.perf_counter()
            sim.solve_cutoff(x, y, z, q, 4e-6)
            t.append(time.perf_counter() - t0)
        return min(t[1:])

    assert seconds(0.01) < 5.0 * seconds(0.0)
