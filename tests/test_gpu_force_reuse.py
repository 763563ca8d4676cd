"""Forces are reused only at the positions they were evaluated at: a query or a
velocity projection at other positions between a force evaluation and a run
leaves no stale forces.  The run equals, bit for bit, that of a context with
the same list and no call in between."""
import numpy as np
import pytest

from geodesic_cuda import amber, backend, synth

pytestmark = pytest.mark.gpu

DT = 0.002


def contexts(precision, constrained):
    atoms, topo, state, _ = synth.generate(600, seed=21, relax_iters=60, h_fraction=0.4 if constrained else 0.0)
    if constrained:
        topo = amber.promote_hydrogen_bonds(topo, atoms)
        assert len(topo.constr_i) > 50
    p = backend.SimParams(box_size=(1000.0,) * 3, r_cutoff=10.0, r_skin=12.0, r_switch=8.0, coulomb=True,
                          precision=precision, max_constr_iter=200, constr_tol=1e-10)
    a = np.ascontiguousarray(state.pos)
    b = a + 0.02 * np.sin(np.arange(a.size)).reshape(a.shape)
    return [backend.CudaBackend(atoms, topo, p) for _ in range(2)], a, np.ascontiguousarray(b), state.vel


@pytest.mark.parametrize("precision", [backend.PRECISION_MIXED, backend.PRECISION_FP64])
@pytest.mark.parametrize("call", ["needs_rebuild", "constrain_velocities"])
@pytest.mark.parametrize("resident", [False, True])
def test_run_after_a_query_at_other_positions(precision, call, resident):
    constrained = call == "constrain_velocities"
    (x, y), a, b, vel = contexts(precision, constrained)
    out = []
    for be, query in ((x, True), (y, False)):
        q, v = a.copy(), np.ascontiguousarray(vel).copy()
        be.build_neighbor_list(q)
        if query:
            be.compute_forces(q)
            if call == "needs_rebuild":
                assert not be.needs_rebuild(b)
            else:
                be.constrain_velocities(b, v)
        elif constrained:
            be.constrain_velocities(b, v)
        q = b.copy()
        if resident:
            be.upload_state(q, v)
            be.run_resident(DT, 3)
            be.synchronize()
            be.download_state(q, v)
        else:
            be.steps(q, v, DT, 3)
        out.append((q, v))
        be.close()
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])


def test_a_query_at_the_same_positions_keeps_the_energy():
    (x, y), a, _, _ = contexts(backend.PRECISION_MIXED, False)
    x.build_neighbor_list(a)
    x.compute_forces(a)
    assert not x.needs_rebuild(a)
    assert x.ensemble_energies()[0][0] == x.potential_energy()
    x.close()
    y.close()
