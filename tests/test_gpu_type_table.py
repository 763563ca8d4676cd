"""Small systems whose pair table is near the 48 KB of shared memory that a
block has without an opt-in (16 bytes per type pair: 54 types leave room for the
block-per-item kernel's own shared memory, 55 fit alone, 56 are read through
L1, 64 are the most): forces of one evaluation against the oracle
(|dF| <= 1e-5 max(|F|, 1) per component), and steps bit for bit against the
kernel-graph form, with and without constraints."""
import numpy as np
import pytest

import oracle
from geodesic_cuda import amber, backend

pytestmark = pytest.mark.gpu

KW = dict(box_size=(1000.0,) * 3, r_cutoff=8.0, r_skin=9.0, r_switch=6.0, coulomb=True)


def system(types, constrained):
    """A jittered lattice, its atoms of `types` (sigma, epsilon) pairs in turn."""
    n = 400
    r = np.random.default_rng(types)
    g = np.stack(np.meshgrid(*[np.arange(8)] * 3, indexing="ij")).reshape(3, -1)[:, :n]
    pos = np.ascontiguousarray((g + 0.5 + r.uniform(-0.05, 0.05, g.shape)) * 3.6)
    k = np.arange(n) % types
    atoms = amber.AtomData(2.8 + 0.005 * k, 0.05 + 0.001 * k, np.full(n, 12.0), r.uniform(-0.1, 0.1, n),
                           np.full(n, 1, np.uint8), np.zeros(n, np.uint32), [])
    t = amber.BondedTopology.empty()
    if constrained:  # pairs of lattice neighbours
        i = np.arange(0, 64, 2)
        t.constr_i, t.constr_j = i.astype(np.uint32), (i + 1).astype(np.uint32)
        d = pos[:, i] - pos[:, i + 1]
        t.constr_dsq = (d * d).sum(0)
        t.excl_i, t.excl_j = t.constr_i.copy(), t.constr_j.copy()
    vel = np.ascontiguousarray(r.standard_normal((3, n)) * 2.0)
    return atoms, t, pos, vel


@pytest.mark.parametrize("types", [1, 54, 55, 56, 64])
def test_forces_match_the_oracle(types):
    atoms, t, pos, _ = system(types, False)
    be = backend.CudaBackend(atoms, t, backend.SimParams(**KW))
    kw = {k: v for k, v in KW.items() if k != "box_size"}
    ob = oracle.CpuBackend(atoms, t, oracle.make_params(box=KW["box_size"], periodic=False, n_threads=1, **kw))
    be.build_neighbor_list(pos)
    ob.build_neighbor_list(pos.copy())
    f, fr = be.compute_forces(pos), ob.compute_forces(pos)
    assert np.max(np.abs(f - fr) / np.maximum(np.abs(fr), 1.0)) <= 1e-5
    be.close()


@pytest.mark.parametrize("constrained", [False, True])
@pytest.mark.parametrize("types", [54, 55, 56, 64])
def test_steps_match_the_kernel_graph(types, constrained):
    atoms, t, pos0, vel0 = system(types, constrained)
    out = []
    for graph in (False, True):
        be = backend.CudaBackend(atoms, t, backend.SimParams(**KW))
        if graph:
            be.step_form(backend.STEP_GRAPH)
        pos, vel = pos0.copy(), vel0.copy()
        be.constrain_velocities(pos, vel)
        for k in (1, 5):
            e, _, f = be.steps(pos, vel, 0.002, k, want_forces=True)
        out.append((pos, vel, f, e))
        be.close()
    for x, y in zip(out[0][:3], out[1][:3]):
        assert np.array_equal(x, y)
    assert out[0][3] == out[1][3]
