"""The potential energy at given positions on one list is the same number
whichever call evaluates it: steps() (whose columns end before the outer half
of the skin while nothing has moved far) and compute_forces() (whole columns),
and a batch's per-system energies after resident steps and after a fresh
evaluation.  Work items of one to many 32-entry chunks."""
import numpy as np
import pytest

from geodesic_cuda import backend, synth

pytestmark = pytest.mark.gpu

P = dict(box_size=(1000.0,) * 3, r_cutoff=10.0, r_skin=13.0, r_switch=8.0, coulomb=True)


@pytest.mark.parametrize("n,split", [(700, 1), (700, 3), (700, 5), (700, 16), (4000, 2), (4000, 7), (20000, 3),
                                     (50000, 0)])
def test_one_system(n, split):
    atoms, topo, state, _ = synth.generate(n, seed=3, relax_iters=40)
    be = backend.CudaBackend(atoms, topo, backend.SimParams(**P))
    if split:
        be.pair_shape(split, 4)
    pos, vel = np.ascontiguousarray(state.pos), np.ascontiguousarray(state.vel)
    be.build_neighbor_list(pos)
    e, rebuilds, f = be.steps(pos, vel, 0.001, 2, want_forces=True)
    assert rebuilds == 0
    f = f.copy()
    assert np.array_equal(be.compute_forces(pos), f)
    assert be.potential_energy() == e
    be.close()


def test_batch():
    sys_ = [synth.generate(n, seed=n, relax_iters=40)[:3] for n in (800, 1500, 300)]
    be = backend.CudaBackend.ensemble([s[0] for s in sys_], [s[1] for s in sys_], backend.SimParams(**P))
    be.pair_shape(2, 4)
    pos = np.ascontiguousarray(np.concatenate([s[2].pos for s in sys_], axis=1))
    vel = np.ascontiguousarray(np.concatenate([s[2].vel for s in sys_], axis=1))
    be.build_neighbor_list(pos)
    be.steps(pos, vel, 0.001, 2)
    e = be.ensemble_energies()[0]
    be.compute_forces(pos)
    assert np.array_equal(be.ensemble_energies()[0], e)
    be.close()
