"""Device memory of a loaded particle set: its own arrays (94 bytes per particle
with a quarter of head room), and the staged positions only for a batch."""
import numpy as np
import pytest

import amk

pytestmark = pytest.mark.gpu


def test_load_reserves_the_particle_arrays_only():
    import torch
    n = 1 << 23
    x = np.zeros(n)
    sp = np.ones(n, np.uint8)
    with amk.Simulation() as s:
        s.set_particles(x[:1000], x[:1000], x[:1000], x[:1000], x[:1000], x[:1000], sp[:1000])
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        s.set_particles(x, x, x, x, x, x, sp)
        torch.cuda.synchronize()
        taken = before - torch.cuda.mem_get_info()[0]
    assert taken < 125 * n, taken / n
