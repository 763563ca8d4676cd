"""Work items of the mixed pair arithmetic at the sizes where they can go
wrong: groups with padding lanes, items without columns (a split larger than
the column has chunks), pairs across the faces of a small box.

Forces: |dF| <= 1e-5 max(|F|, 1) per component against the oracle, and the
same bits for every split.  Energy: each pair's FP32 value carries a few
roundings and is summed in FP32 over a chunk, so |dE| is within 32 * 2^-24 of
the sum of the pair energies' magnitudes (16 roundings a term, both halves of
the list); the bonded terms are FP64."""
import numpy as np
import pytest

import oracle
from geodesic_cuda import amber, backend, synth

pytestmark = pytest.mark.gpu

RC, RL, RSW = 10.0, 12.0, 8.0
KC = 332.0522173


def magnitude(atoms, topo, pos, box):
    """Sum of |V| over the pairs inside the cutoff (unswitched: an upper bound)."""
    d = pos[:, :, None] - pos[:, None, :]
    if box:
        d -= box * np.round(d / box)
    r = np.sqrt((d * d).sum(0))
    iu = np.triu_indices(pos.shape[1], 1)
    excl = {(min(a, b), max(a, b)) for a, b in zip(topo.excl_i.tolist(), topo.excl_j.tolist())}
    total = 0.0
    for i, j in zip(*iu):
        if r[i, j] <= RC and (i, j) not in excl:
            s6 = (0.5 * (atoms.sigma[i] + atoms.sigma[j]) / r[i, j]) ** 6
            e = np.sqrt(atoms.epsilon[i] * atoms.epsilon[j])
            total += 4 * e * s6 * (s6 + 1) + KC * abs(atoms.charge[i] * atoms.charge[j]) / r[i, j]
    return total


@pytest.mark.parametrize("n,box", [(1, None), (2, None), (31, None), (32, None), (33, None), (40, None), (75, None),
                                   (375, None), (97, 24.5), (375, 25.0), (700, 31.0)])
def test_pair_items_match_the_oracle_for_every_split(n, box):
    if n <= 2:
        t = amber.BondedTopology.empty()
        atoms = amber.AtomData(np.full(n, 3.0), np.full(n, 0.1), np.full(n, 12.0), np.linspace(-0.3, 0.4, n),
                               np.full(n, 1, np.uint8), np.zeros(n, np.uint32), [])
        pos = np.ascontiguousarray(np.array([[1.0, 4.1], [2.0, 2.5], [3.0, 3.2]])[:, :n])
    else:
        atoms, t, state, _ = synth.generate(n, seed=77 + n, relax_iters=60)
        pos = np.ascontiguousarray(state.pos)
    kw = dict(r_cutoff=RC, r_skin=RL, r_switch=RSW, coulomb=True)
    size = (box,) * 3 if box else (1000.0,) * 3
    p = backend.SimParams(box_size=size, periodic=box is not None, **kw)
    if box:  # the droplet across the faces of the box
        t = amber.BondedTopology.empty()
        pos = np.ascontiguousarray(pos - pos.mean(axis=1, keepdims=True))
    be = backend.CudaBackend(atoms, t, p)
    ob = oracle.CpuBackend(atoms, t, oracle.make_params(box=size, periodic=box is not None, n_threads=1, **kw))
    pg, pr = pos.copy(), pos.copy()
    be.build_neighbor_list(pg)
    ob.build_neighbor_list(pr)
    f0 = be.compute_forces(pg).copy()
    e0 = be.potential_energy()
    fr = ob.compute_forces(pr)
    assert np.max(np.abs(f0 - fr) / np.maximum(np.abs(fr), 1.0)) <= 1e-5
    assert abs(e0 - ob.potential_energy) <= 32 * 2.0 ** -24 * magnitude(atoms, t, pg, box) + 1e-9 * abs(ob.potential_energy)
    for split in (1, 3, 7, 16):
        be.pair_shape(split, 4)
        assert np.array_equal(be.compute_forces(pg), f0), split
    be.step_form(backend.STEP_GRAPH)
    assert np.array_equal(be.compute_forces(pg), f0)
    be.close()
