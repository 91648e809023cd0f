"""Contact search of a batch through its hashed cells: cell sizes set by the
grid and by the contact radius, one cell for all, particles that leave the
grid, species without a partner. Instances must annihilate exactly as each
does in a context of its own (same streams, same pairs)."""
import numpy as np
import pytest

import amk
from test_gpu_batch import alone, assert_same, instance, load, sliced

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("radius,sigma,vel", [
    (2e-7, 1e-5, 1e2),    # cells set by the grid, far larger than the radius
    (1.5e-5, 1e-4, 2e4),  # cells of the radius, about one particle each
    (4e-5, 1e-4, 2e4),    # dozens of candidates
    (1e-2, 1e-4, 2e4),    # every particle in one cell
    (3e-5, 1e-4, 5e6),    # particles leave the grid within a step or two
])
def test_contacts_as_in_single_contexts(radius, sigma, vel):
    insts = [instance(n, 40 + k, pair=pair, sigma=sigma, vel=vel, contact_radius=radius, coulomb_forces_enabled=0)
             for k, (n, pair) in enumerate([(1, ("positron", "electron")), (301, ("positron", "electron")),
                                            (700, ("antiproton", "proton")), (128, ("positron", "antiproton")),
                                            (1500, ("electron", "positron"))])]
    with amk.Simulation(insts[0][3]) as s:
        offs = load(s, insts)
        s.batch_step(3)
        st = s.get_particles()
    for k, inst in enumerate(insts):
        assert_same(sliced(st, offs[k], offs[k + 1]), alone(inst, 3))
    if radius > 1e-6 and vel < 1e6:
        assert not st["alive"].all()
