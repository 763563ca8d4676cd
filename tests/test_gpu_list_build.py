"""The list build where its sweep changes: pair sets bit-exact against the
oracle (the reference's FP64 list test) for padding lanes, boxes so small that
a whole dimension is scanned or a pair's image differs from its group's,
surface groups whose rows share a sweep, more than eight exclusions on an atom
(one of them far away), and both sides of the split into y rows."""
import numpy as np
import pytest

import oracle
from geodesic_cuda import amber, backend, synth

pytestmark = pytest.mark.gpu


def gas(n, box, seed):
    r = np.random.default_rng(seed)
    k = int(np.ceil(n ** (1 / 3)))
    g = np.stack(np.meshgrid(*[np.arange(k)] * 3, indexing="ij")).reshape(3, -1)[:, :n]
    return np.ascontiguousarray((g + 0.5 + r.uniform(-0.3, 0.3, g.shape)) * (box / k))


def shapes(name, n):
    r = np.random.default_rng(n)
    if name == "droplet":
        p = r.standard_normal((3, 4 * n))
        p = p / np.linalg.norm(p, axis=0) * r.uniform(0, 1, 4 * n) ** (1 / 3) * (n / 0.08 * 3 / (4 * np.pi)) ** (1 / 3)
        return np.ascontiguousarray(p[:, :n])
    if name == "sheet":  # a thin layer: short rows in every cell layer
        e = (n / 0.3) ** 0.5
        return np.ascontiguousarray(np.stack([r.uniform(0, e, n), r.uniform(0, 3, n), r.uniform(0, e, n)]))
    p = gas(n, (n / 0.1) ** (1 / 3), n)  # a droplet and far outliers, beyond the grid's core
    p[:, ::97] += r.uniform(-400, 400, p[:, ::97].shape)
    return np.ascontiguousarray(p)


@pytest.mark.parametrize("n,box,shape,r_list", [
    (1, None, "droplet", 12.0), (33, None, "droplet", 12.0), (1000, None, "droplet", 12.0),
    (700, None, "sheet", 12.0), (2100, None, "outliers", 12.0), (9599, None, "droplet", 9.0), (9700, None, "droplet", 9.0),
    (97, 13.1, None, 6.5), (500, 24.1, None, 12.0), (1536, 24.9, None, 12.0), (3001, 30.2, None, 12.0),
    (3500, 36.5, None, 12.0), (9700, 50.0, None, 8.0)])
def test_pairs_equal_the_oracles(n, box, shape, r_list):
    pos = shapes(shape, n) if shape else gas(n, box, n)
    t = amber.BondedTopology.empty()
    r = np.random.default_rng(5)
    if n > 30:
        # atom 7 excludes 20 others, near and far; a sprinkle of pairs besides
        ei = np.concatenate([np.full(20, 7), r.integers(0, n, n // 3)])
        ej = np.concatenate([r.permutation(n)[:20], r.integers(0, n, n // 3)])
        t.excl_i, t.excl_j = ei[ei != ej].astype(np.uint32), ej[ei != ej].astype(np.uint32)
    atoms = amber.AtomData(np.full(n, 3.0), np.full(n, 0.1), np.full(n, 12.0), np.zeros(n), np.full(n, 1, np.uint8),
                           np.zeros(n, np.uint32), [])
    size = (box,) * 3 if box else (10000.0,) * 3
    kw = dict(r_cutoff=0.8 * r_list, r_skin=r_list, r_switch=0.6 * r_list)
    be = backend.CudaBackend(atoms, t, backend.SimParams(box_size=size, periodic=box is not None, **kw))
    ob = oracle.CpuBackend(atoms, t, oracle.make_params(box=size, periodic=box is not None, n_threads=8, **kw))
    pg, pr = pos.copy(), pos.copy()
    be.build_neighbor_list(pg)
    ob.build_neighbor_list(pr)
    assert np.array_equal(pg, pr)
    (gi, gj), (ri, rj) = be.pairs(), ob.pairs()
    assert len(gi) == len(ri) and np.array_equal(gi, ri) and np.array_equal(gj, rj)
    be.close()


@pytest.mark.parametrize("n,box,skin,steps", [(700, 45.0, 10.3, 190), (3200, 75.0, 10.5, 130)])
def test_rebuilds_of_a_run_that_outgrow_the_staging_area(n, box, skin, steps):
    """A droplet that condenses in a large periodic box: the staging area is
    sized by the mean density and the first lists, and a resident run cannot
    grow it.  The run ends, and the forces at its end are a fresh context's:
    |dF| <= 1e-5 max(|F|, 1) per component."""
    atoms, topo, state, _ = synth.generate(n, seed=11 + n, relax_iters=60)
    pos = np.ascontiguousarray(state.pos - state.pos.mean(axis=1, keepdims=True))
    vel = np.ascontiguousarray(state.vel).copy()
    p = backend.SimParams(box_size=(box,) * 3, periodic=True, r_cutoff=10.0, r_skin=skin, r_switch=8.0, coulomb=True,
                          bonded_min_image=True)
    be = backend.CudaBackend(atoms, topo, p)
    first = 0
    for k in (3, 10, steps // 2, steps // 2):
        _, _, f = be.steps(pos, vel, 0.002, k, first_step=first, want_forces=True)
        first += k
        other = backend.CudaBackend(atoms, topo, p)
        q = pos.copy()
        other.build_neighbor_list(q)
        fr = other.compute_forces(q)
        other.close()
        assert np.max(np.abs(f - fr) / np.maximum(np.abs(fr), 1.0)) <= 1e-5, first
    be.close()


def test_wrap_at_the_faces():
    """The wrap into the box is x - L floor(x / L) in FP64, bit for bit, at and
    around the faces and the zeros."""
    L = 40.0
    x = np.array([0.0, -0.0, 5e-324, -5e-324, -1e-17, 1e-17, L, np.nextafter(L, 0), np.nextafter(L, 99), -L, 2 * L,
                  np.nextafter(2 * L, 0), 3.25, -3.25, 97.5, -1e6 / 3])
    n = 3 * len(x)
    pos = np.stack([np.linspace(1, 39, n)] * 3)
    for d in range(3):  # each value in each component, the atoms apart in another
        pos[d, d * len(x):(d + 1) * len(x)] = x
    pos = np.ascontiguousarray(pos)
    atoms = amber.AtomData(np.full(n, 3.0), np.full(n, 0.1), np.full(n, 12.0), np.zeros(n), np.full(n, 1, np.uint8),
                           np.zeros(n, np.uint32), [])
    p = backend.SimParams(box_size=(L,) * 3, periodic=True, r_cutoff=8.0, r_skin=10.0, r_switch=7.0)
    be = backend.CudaBackend(atoms, amber.BondedTopology.empty(), p)
    want = pos - L * np.floor(pos / L)
    be.build_neighbor_list(pos)
    be.close()
    assert np.array_equal(pos.view(np.uint64), want.view(np.uint64))
