"""A build wraps the positions once, x - L floor(x / L) in FP64 bit for bit,
also where the list has to grow and be built again: a coordinate that the wrap
puts on the face L stays there.  A resident run's rebuild that outgrows the
list, of a single system and of one system of a batch whose other system is
built again without having moved."""
import numpy as np
import pytest

from geodesic_cuda import amber, backend

pytestmark = pytest.mark.gpu

L, N = 60.0, 1500
P = dict(box_size=(L,) * 3, periodic=True, r_cutoff=8.0, r_skin=10.0, r_switch=7.0)


def inert(n):
    return amber.AtomData(np.zeros(n), np.zeros(n), np.full(n, 12.0), np.zeros(n), np.full(n, 1, np.uint8),
                          np.zeros(n, np.uint32), [])


def scattered(seed):
    return np.random.default_rng(seed).uniform(0.5, L - 0.5, (3, N))


def dense(seed):
    """A blob of a few angstroms in the middle of the box, an atom of it past each lower face."""
    pos = L / 2 + np.random.default_rng(seed).uniform(-6, 6, (3, N))
    for d in range(3):
        pos[d, d] = -1e-17
    pos[:, 3] = [-1.0, L + 2.5, np.nextafter(L, 99)]
    return np.ascontiguousarray(pos)


def wrapped(pos):
    return pos - L * np.floor(pos / L)


@pytest.mark.parametrize("precision", [backend.PRECISION_MIXED, backend.PRECISION_FP64])
@pytest.mark.parametrize("first", [0, 1])
def test_batch(precision, first):
    sys_ = [(inert(N), amber.BondedTopology.empty())] * 2
    be = backend.CudaBackend.ensemble([s[0] for s in sys_], [s[1] for s in sys_],
                                      backend.SimParams(precision=precision, **P))
    q = np.concatenate([scattered(1), scattered(2)], axis=1)
    q[0, 5] = q[0, N + 5] = -1e-17
    be.build_neighbor_list(q)
    assert q[0, 5] == L and q[0, N + 5] == L
    cap = be.counters()["cap"]
    moved = slice(first * N, (first + 1) * N)
    still = slice((1 - first) * N, (2 - first) * N)
    q[:, moved] = dense(3)
    want = q.copy()
    want[:, moved] = wrapped(q[:, moved])
    # the other system is built again too, at positions inside the box already;
    # its coordinate on the face is wrapped once more, as a build of it does
    want[:, still] = wrapped(q[:, still])
    vel = np.zeros_like(q)
    be.upload_state(q, vel)
    be.forces_resident()
    assert be.counters()["cap"] > cap
    got = np.zeros_like(q)
    be.download_state(got, vel)
    be.close()
    assert np.array_equal(got.view(np.uint64), want.view(np.uint64))


@pytest.mark.parametrize("precision", [backend.PRECISION_MIXED, backend.PRECISION_FP64])
def test_single_system(precision):
    be = backend.CudaBackend(inert(N), amber.BondedTopology.empty(), backend.SimParams(precision=precision, **P))
    q = scattered(1)
    be.build_neighbor_list(q)
    cap = be.counters()["cap"]
    q = dense(2)
    vel = np.zeros_like(q)
    got = q.copy()
    be.upload_state(got, vel)
    be.forces_resident()
    assert be.counters()["cap"] > cap
    be.download_state(got, vel)
    be.close()
    assert np.array_equal(got.view(np.uint64), wrapped(q).view(np.uint64))
