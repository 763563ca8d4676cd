"""Pairs without Lennard-Jones well and charge almost in contact exert no force
in the FP64 path (force/nonbonded.rs:20-82 evaluates the term only where
epsilon is not 0), at any distance down to where (sigma / r)^12 overflows; a
third atom's pairs with them are unchanged."""
import numpy as np
import pytest

from geodesic_cuda import amber, backend

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("r", [0.0, 1e-120, 1e-60, 1e-25, 1e-3])
def test_no_force_without_a_well(r):
    atoms = amber.AtomData(np.array([3.0, 3.0, 3.4]), np.array([0.0, 0.0, 0.2]), np.full(3, 12.0),
                           np.array([0.0, 0.0, 0.3]), np.full(3, 1, np.uint8), np.zeros(3, np.uint32), [])
    pos = np.ascontiguousarray([[0.0, r, 3.0], [0.0, 0.0, 1.0], [0.0, 0.0, 2.0]])
    be = backend.CudaBackend(atoms, amber.BondedTopology.empty(),
                             backend.SimParams(box_size=(1000.0,) * 3, r_cutoff=10.0, r_skin=12.0, r_switch=8.0,
                                               coulomb=True, precision=backend.PRECISION_FP64))
    be.build_neighbor_list(pos)
    f = be.compute_forces(pos)
    assert np.array_equal(f, np.zeros((3, 3))) and be.potential_energy() == 0.0
    be.close()
