"""The constrained resident step (two cooperative launches, a constraint per
lane) against the trait's calls one by one (separate launches): positions,
velocities and energy bit for bit, for stars of 1 to 8 constraints in counts
around the warps' edges, with and without other atoms, and the same failure
when the solver does not converge."""
import numpy as np
import pytest

from geodesic_cuda import amber, backend

pytestmark = pytest.mark.gpu

DT = 0.002


def system(sizes, n_free, seed):
    """Stars of the given sizes on a lattice, centre first or last in caller order, and free atoms."""
    r = np.random.default_rng(seed)
    total = len(sizes) + n_free
    k = int(np.ceil(total ** (1 / 3)))
    sites = (np.stack(np.meshgrid(*[np.arange(k)] * 3, indexing="ij")).reshape(3, -1)[:, :total] + 0.5) * 4.5
    sites = sites[:, r.permutation(total)]
    pos, mass, el, ci, cj, ei, ej = [], [], [], [], [], [], []
    for s, nc in enumerate(sizes):
        d = r.standard_normal((3, nc))
        # spread the hydrogens so that no two coincide
        d = d / np.linalg.norm(d, axis=0) + 1e-3 * r.standard_normal((3, nc))
        d = d / np.linalg.norm(d, axis=0) * 1.09
        atoms = np.concatenate([sites[:, s:s + 1], sites[:, s:s + 1] + d], axis=1)
        base, cen_last = sum(p.shape[1] for p in pos), bool(r.integers(2))
        if cen_last:
            atoms = atoms[:, ::-1]
        cen = base + (nc if cen_last else 0)
        hs = [base + q for q in range(nc + 1) if base + q != cen]
        for h in hs:
            a, b = (cen, h) if r.integers(2) else (h, cen)
            ci.append(a)
            cj.append(b)
        u, w = np.triu_indices(nc + 1, 1)  # a star's atoms exclude each other
        ei.append(base + u)
        ej.append(base + w)
        m = np.full(nc + 1, 1.008)
        m[cen - base] = 12.0 + r.uniform()
        pos.append(atoms)
        mass.append(m)
        el.append((m > 2).astype(np.uint8))
    pos.append(sites[:, len(sizes):])
    mass.append(np.full(n_free, 14.0))
    el.append(np.full(n_free, 1, np.uint8))
    pos, mass = np.ascontiguousarray(np.concatenate(pos, axis=1)), np.concatenate(mass)
    n = len(mass)
    t = amber.BondedTopology.empty()
    order = r.permutation(len(ci))
    t.constr_i, t.constr_j = np.array(ci, np.uint32)[order], np.array(cj, np.uint32)[order]
    t.constr_dsq = np.full(len(ci), 1.09 ** 2)
    t.excl_i, t.excl_j = np.concatenate(ei).astype(np.uint32), np.concatenate(ej).astype(np.uint32)
    atoms = amber.AtomData(np.full(n, 2.0), np.full(n, 0.02), mass, r.uniform(-0.05, 0.05, n), np.concatenate(el),
                           np.zeros(n, np.uint32), [])
    vel = r.standard_normal((3, n)) * np.sqrt(0.0019872041 * 300.0 * 20.455 ** 2 / mass)
    return atoms, t, pos, np.ascontiguousarray(vel)


CASES = [([1], 0), ([2] * 5, 3), ([1] * 33, 100), ([3] * 9 + [4] * 8, 1), ([8] * 4 + [5, 6, 7], 40),
         ([1] * 31 + [2] * 17 + [3] * 8 + [4] * 2 + [5] * 3 + [8], 700),
         # one star past a warp per scheduler with four lanes a constraint (152 SMs), and the last at it
         ([2] * 2432, 5), ([2] * 2433, 5)]


@pytest.mark.parametrize("precision", [backend.PRECISION_MIXED, backend.PRECISION_FP64])
@pytest.mark.parametrize("sizes,n_free", CASES)
def test_resident_steps_equal_the_traits_calls(sizes, n_free, precision):
    atoms, t, pos, vel = system(sizes, n_free, 11)
    p = backend.SimParams(box_size=(1000.0,) * 3, r_cutoff=8.0, r_skin=9.0, r_switch=6.0, coulomb=True,
                          precision=precision, max_constr_iter=200)
    a, b = backend.CudaBackend(atoms, t, p), backend.CudaBackend(atoms, t, p)
    pa, va, pb, vb = pos.copy(), vel.copy(), pos.copy(), vel.copy()
    for be, q, v in ((a, pa, va), (b, pb, vb)):
        be.build_neighbor_list(q)
        be.constrain_velocities(q, v)
    assert np.array_equal(va, vb)
    f = b.compute_forces(pb)
    rebuilds = 0
    for n_steps in (1, 7, 12):
        e, nr, _ = a.steps(pa, va, DT, n_steps)
        rebuilds += nr
        for _ in range(n_steps):
            b.half_kick(vb, f, DT / 2)
            b.geodesic_drift(pb, vb, DT)
            if b.needs_rebuild(pb):
                b.build_neighbor_list(pb)
            f = b.compute_forces(pb)
            b.half_kick(vb, f, DT / 2)
            b.constrain_velocities(pb, vb)
        assert np.array_equal(pa, pb) and np.array_equal(va, vb)
        assert e == b.potential_energy()
    a.close()
    b.close()


def test_a_failed_projection_is_the_traits():
    atoms, t, pos, vel = system([1] * 40 + [3] * 20 + [6] * 3, 50, 5)
    # three iterations: the singles converge, some of the larger stars do not
    p = backend.SimParams(box_size=(1000.0,) * 3, r_cutoff=8.0, r_skin=9.0, r_switch=6.0, max_constr_iter=3)
    a, b = backend.CudaBackend(atoms, t, p), backend.CudaBackend(atoms, t, p)
    pa, va, pb, vb = pos.copy(), vel.copy(), pos.copy(), vel.copy()
    a.build_neighbor_list(pa)
    b.build_neighbor_list(pb)
    f = b.compute_forces(pb)
    with pytest.raises(backend.ConvergenceError) as ea:
        a.steps(pa, va, DT, 1, first_step=9)
    b.half_kick(vb, f, DT / 2)
    with pytest.raises(backend.ConvergenceError) as eb:
        b.geodesic_drift(pb, vb, DT, step=9)
    for k in ("step", "constraint_idx", "atom_i", "atom_j"):
        assert getattr(ea.value, k) == getattr(eb.value, k), k
    # the caller's state as the projection left it, and a context that works on
    assert np.array_equal(pa, pb) and np.array_equal(va, vb)
    a.close()
    b.close()
