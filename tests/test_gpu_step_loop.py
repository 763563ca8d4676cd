"""Launches that run several steps (small systems in the persistent step form)
against the kernel-graph form, one launch sequence a step: the same positions,
velocities, forces and rebuild counts, bit for bit, for calls shorter than a
launch's step limit (64), at it, one past it and several launches long, and
with rebuilds that end a launch early."""
import numpy as np
import pytest

from geodesic_cuda import backend, synth

pytestmark = pytest.mark.gpu

DT = 0.002
CALLS = (1, 2, 63, 64, 65, 130)


@pytest.mark.parametrize("n,box,skin", [(33, None, 12.0), (224, None, 10.2), (224, None, 12.0), (700, None, 10.3),
                                        (700, 45.0, 12.0), (3200, None, 10.5), (3201, None, 12.0)])
def test_calls_of_any_length_match_the_kernel_graph(n, box, skin):
    atoms, topo, state, _ = synth.generate(n, seed=11 + n, relax_iters=60)
    pos0 = np.ascontiguousarray(state.pos)
    if box:  # the droplet across the faces of the box
        pos0 = np.ascontiguousarray(pos0 - pos0.mean(axis=1, keepdims=True))
    p = backend.SimParams(box_size=(box or 1000.0,) * 3, periodic=box is not None, r_cutoff=10.0, r_skin=skin,
                          r_switch=8.0, coulomb=True, bonded_min_image=box is not None)
    runs = []
    for form in (backend.STEP_PERSISTENT, backend.STEP_GRAPH):
        be = backend.CudaBackend(atoms, topo, p)
        be.step_form(form)
        pos, vel = pos0.copy(), np.ascontiguousarray(state.vel).copy()
        out, step = [], 0
        for k in CALLS:
            e, rebuilds, f = be.steps(pos, vel, DT, k, first_step=step, want_forces=True)
            step += k
            out.append((pos.copy(), vel.copy(), f, e, rebuilds))
        runs.append(out)
        be.close()
    for k, a, b in zip(CALLS, *runs):
        for x, y in zip(a[:3], b[:3]):
            assert np.array_equal(x.view(np.uint64), y.view(np.uint64)), k
        assert a[3:] == b[3:], k
    if skin < 11.0:  # rebuilds cut launches short
        assert sum(r[4] for r in runs[0]) >= 2
