"""List builds of a batch on both sides of the row split: a build of every
system (all groups together past 300) and a rebuild of some of them (few enough
to split a layer's rows over warps) give the oracle's pairs, and forces bit for
bit those of each system alone."""
import numpy as np
import pytest

import oracle
from geodesic_cuda import backend, synth

pytestmark = pytest.mark.gpu

KW = dict(r_cutoff=10.0, r_skin=12.0, r_switch=8.0)
SIZES = (700, 2100, 33, 3000, 2, 1500, 2999)  # 326 groups


def test_builds_of_every_and_of_some_systems():
    sys_ = [synth.generate(n, seed=n, relax_iters=20)[:3] for n in SIZES]
    p = backend.SimParams(box_size=(1000.0,) * 3, coulomb=True, **KW)
    op = oracle.make_params(box=p.box_size, periodic=False, n_threads=4, **KW)
    be = backend.CudaBackend.ensemble([s[0] for s in sys_], [s[1] for s in sys_], p)
    off = be.offsets
    pos = np.ascontiguousarray(np.concatenate([s[2].pos for s in sys_], axis=1))
    be.build_neighbor_list(pos)
    vel = np.zeros_like(pos)
    r = np.random.default_rng(3)
    for moved in ((), (1,), (2, 3, 4), (0, 6)):
        for k in moved:
            # every atom of the system past half the skin
            pos[:, off[k]:off[k + 1]] = 5.0 + pos[:, off[k]:off[k + 1]] * (1.0 + 0.1 * r.random())
        be.upload_state(pos, vel)
        be.forces_resident()
        gi, gj = be.pairs()
        f = be.compute_forces(pos).copy()
        for k, (atoms, topo, _) in enumerate(sys_):
            q = np.ascontiguousarray(pos[:, off[k]:off[k + 1]])
            mine = (gi >= off[k]) & (gi < off[k + 1])
            if k in moved or not moved:
                ri, rj = oracle.neighbor_build(q.copy(), atoms, topo, op, cells=True)
                assert np.array_equal(gi[mine] - off[k], ri) and np.array_equal(gj[mine] - off[k], rj), (moved, k)
                one = backend.CudaBackend(atoms, topo, p)
                one.build_neighbor_list(q)
                assert np.array_equal(one.compute_forces(q), f[:, off[k]:off[k + 1]]), (moved, k)
                one.close()
    assert be.counters()["rebuilds"] == len(SIZES) + 6
    be.close()
