"""Graph chunks of a batch between calls that grow the context's scratch (its
sorts, scans and cutoff solver work there): the steps must not depend on what
the context did in between, nor on which kind of step came first."""
import numpy as np
import pytest

import amk
from test_gpu_batch import assert_same, instance, load

pytestmark = pytest.mark.gpu


def _grow(s, what):
    rng = np.random.default_rng(9)
    x, y, z = rng.normal(0.0, 1e-4, (3, 60000))
    q = np.full(60000, 1.6e-19)
    if what == "energy":  # cutoff energies: the cell counters of the largest instance
        s.batch_energy()
    elif what == "cutoff":
        s.solve_cutoff(x, y, z, q, 1e-6)
    elif what == "fmm":
        s.solve_fmm(x, y, z, q, 2, 0.6)
    elif what == "tree":
        s.solve_barnes_hut(x, y, z, q, 0.9)


@pytest.mark.parametrize("method", ["allpairs", "standard"])
@pytest.mark.parametrize("what", ["energy", "cutoff", "fmm", "tree"])
def test_chunks_after_scratch_has_grown(method, what):
    insts = [instance(17000, 61, coulomb_method=method, cutoff_radius=2e-6, contact_radius=1e-6),
             instance(800, 62, coulomb_method=method, contact_radius=1e-6)]
    with amk.Simulation() as s:
        load(s, insts)
        s.batch_step(12)
        plain = s.get_particles()
    with amk.Simulation() as s:
        load(s, insts)
        assert s.batch_info()["graphable"]
        s.batch_step(5, graph_chunk=2)
        _grow(s, what)
        s.batch_step(4, graph_chunk=2)
        _grow(s, what)  # nothing grows: the capture may stay
        s.batch_step(3, graph_chunk=2)
        assert s.step_count() == 12
        got = s.get_particles()
    assert_same(plain, got)


def test_chunks_after_a_serial_step():
    # a serial step leaves the scratch of a batched one unreserved
    insts = [instance(17000, 71, coulomb_forces_enabled=0), instance(900, 72, coulomb_forces_enabled=0)]
    with amk.Simulation() as s:
        load(s, insts)
        s.batch_step(7)
        plain = s.get_particles()
    with amk.Simulation() as s:
        load(s, insts)
        s.batch_step(1, serial=True)
        s.batch_step(6, graph_chunk=2)
        got = s.get_particles()
    assert_same(plain, got)
