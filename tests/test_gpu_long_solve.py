"""A solver that is allowed very many iterations and does not converge ends with
the trait's convergence error, not with a barrier's time limit: the resident
step against the trait's calls one by one (an unreachable tolerance; 1,000,000
iterations, a few seconds)."""
import numpy as np
import pytest

from geodesic_cuda import backend
from test_gpu_constrained_step import DT, system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("iterations", [300, 1_000_000])
def test_a_long_solves_failure_is_the_traits(iterations):
    atoms, t, pos, vel = system([1] * 64, 300, 11)
    p = backend.SimParams(box_size=(1000.0,) * 3, r_cutoff=8.0, r_skin=9.0, r_switch=6.0, constr_tol=1e-300,
                          max_constr_iter=iterations)
    a, b = backend.CudaBackend(atoms, t, p), backend.CudaBackend(atoms, t, p)
    pa, va, pb, vb = pos.copy(), vel.copy(), pos.copy(), vel.copy()
    a.build_neighbor_list(pa)
    b.build_neighbor_list(pb)
    f = b.compute_forces(pb)
    with pytest.raises(backend.ConvergenceError) as ea:
        a.steps(pa, va, DT, 1)
    b.half_kick(vb, f, DT / 2)
    with pytest.raises(backend.ConvergenceError) as eb:
        b.geodesic_drift(pb, vb, DT)
    for k in ("step", "constraint_idx", "atom_i", "atom_j"):
        assert getattr(ea.value, k) == getattr(eb.value, k), k
    assert np.array_equal(pa, pb) and np.array_equal(va, vb)
    a.close()
    b.close()
