"""Groups whose staged words outgrow the staging area are built by the second
kernel: pair lists bit-exact against the oracle for a dense blob that a resident
call finds dispersed (a group's 32 atoms then lie in many short rows of cells,
while the staging area was sized by the blob's build and, with an atom far off,
by a low mean density).  With and without a
periodic box, both sides of the split into y rows (300 groups), alone and in
batches whose other system keeps its list."""
import numpy as np
import pytest

import oracle
from geodesic_cuda import amber, backend

pytestmark = pytest.mark.gpu

KW = dict(r_cutoff=9.0, r_skin=12.0, r_switch=7.0)


def inert(n):
    return amber.AtomData(np.zeros(n), np.zeros(n), np.full(n, 12.0), np.zeros(n), np.full(n, 1, np.uint8),
                          np.zeros(n, np.uint32), [])


def blob(n, centre, seed):
    """A jittered cubic lattice at 0.02 atoms per cubic angstrom and one atom far from it."""
    k = int(np.ceil(n ** (1 / 3)))
    g = np.stack(np.meshgrid(*[np.arange(k)] * 3, indexing="ij")).reshape(3, -1)[:, :n]
    pos = (g - k / 2 + np.random.default_rng(seed).uniform(-0.3, 0.3, g.shape)) * 0.02 ** (-1 / 3) + centre
    pos[:, -1] = centre + 130.0
    return pos


@pytest.mark.parametrize("sizes,box,edge", [((2000,), None, 250.0), ((12000,), None, 500.0), ((2000,), 300.0, 290.0),
                                            ((9700,), 500.0, 499.0), ((2000, 3000), None, 250.0),
                                            ((12000, 9000), None, 500.0)])
def test_pairs_of_a_dispersed_blob(sizes, box, edge):
    centre = box / 2 if box else 1000.0
    p = backend.SimParams(box_size=(box or 10000.0,) * 3, periodic=box is not None, **KW)
    sys_ = [(inert(n), amber.BondedTopology.empty()) for n in sizes]
    be = (backend.CudaBackend(*sys_[0], p) if len(sizes) == 1 else
          backend.CudaBackend.ensemble([s[0] for s in sys_], [s[1] for s in sys_], p))
    parts = [blob(n, centre, k) for k, n in enumerate(sizes)]
    pos = np.ascontiguousarray(np.concatenate(parts, axis=1))
    be.build_neighbor_list(pos)
    n0 = sizes[0]
    pos[:, :n0] = centre + edge * (np.random.default_rng(9).random((3, n0)) - 0.5)
    vel = np.zeros_like(pos)
    be.upload_state(pos, vel)
    be.forces_resident()
    assert be.counters()["rebuilds"] == len(sizes) + 1
    gi, gj = be.pairs()
    be.close()
    op = oracle.make_params(box=p.box_size, periodic=box is not None, n_threads=8, **KW)
    want, first = [], 0
    for n, (atoms, topo) in zip(sizes, sys_):
        ri, rj = oracle.neighbor_build(np.ascontiguousarray(pos[:, first:first + n]), atoms, topo, op, cells=True)
        want.append((ri.astype(np.int64) + first, rj.astype(np.int64) + first))
        first += n
    ri, rj = np.concatenate([w[0] for w in want]), np.concatenate([w[1] for w in want])
    assert len(gi) == len(ri) > n0 / 8
    assert np.array_equal(gi, ri) and np.array_equal(gj, rj)
