"""The launch shape that a context starts with is in the range that gm_pair_shape
accepts and among the shapes that gm_autotune times: a fresh context's split can
be set back, and a split that is not on the tuner's own list is timed too."""
import numpy as np
import pytest

from geodesic_cuda import backend, synth

pytestmark = pytest.mark.gpu

P = dict(box_size=(1000.0,) * 3, r_cutoff=10.0, r_skin=12.0, r_switch=8.0, coulomb=True)
LIST = 8 * 3 * 5  # splits x warps per block x grids


@pytest.mark.parametrize("precision", [backend.PRECISION_MIXED, backend.PRECISION_FP64])
@pytest.mark.parametrize("n", [40, 3200, 8000, 50000])
def test_a_fresh_contexts_split_can_be_set(n, precision):
    atoms, topo, state, _ = synth.generate(n, seed=4, relax_iters=20)
    be = backend.CudaBackend(atoms, topo, backend.SimParams(precision=precision, **P))
    pos = np.ascontiguousarray(state.pos)
    be.build_neighbor_list(pos)
    split = be.counters()["split"]
    f = be.compute_forces(pos).copy()
    e = be.potential_energy()
    be.pair_shape(3, 2)
    assert np.array_equal(be.compute_forces(pos), f)
    be.pair_shape(split, 4)
    assert be.counters()["split"] == split
    assert np.array_equal(be.compute_forces(pos), f) and be.potential_energy() == e
    be.close()


@pytest.mark.parametrize("precision", [backend.PRECISION_MIXED, backend.PRECISION_FP64])
@pytest.mark.parametrize("split,more", [(16, 0), (5, 1)])
def test_the_tuner_times_the_present_split(precision, split, more):
    atoms, topo, state, _ = synth.generate(2000, seed=4, relax_iters=20)
    be = backend.CudaBackend(atoms, topo, backend.SimParams(precision=precision, **P))
    be.step_form(backend.STEP_GRAPH) if precision == backend.PRECISION_MIXED else None
    pos = np.ascontiguousarray(state.pos)
    be.build_neighbor_list(pos)
    be.pair_shape(split, 4)
    be.compute_forces(pos)
    before = be.counters()["launches"]
    choice = be.autotune(reps=1)
    timed = (be.counters()["launches"] - before) // 2  # a warm-up and a timed launch each
    assert timed // 15 == 8 + more
    be.pair_shape(choice["split"], choice["warps_per_block"], choice["grid"])
    be.close()
