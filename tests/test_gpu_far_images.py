"""Forces at positions that are whole boxes away from where the list was built
(a caller that keeps its trajectory unwrapped): those of the wrapped positions.

The FP64 path's forces differ by the rounding of the shifted coordinates alone:
at k boxes of 46.4 A a coordinate and the product L k are within 2^-53 k L each,
so a pair's difference is within 4 * 2^-53 k L = 2.1e-14 k of the wrapped one;
a force component sums ~30 close neighbours of at most 100 kcal/mol/A^2 each:
|dF| <= 6.2e-11 k, and 1e-9 for the wrapped positions' own rounding."""
import numpy as np
import pytest

from geodesic_cuda import amber, backend

pytestmark = pytest.mark.gpu

L = 46.4


@pytest.mark.parametrize("k", [1, 2, 3, 40, 3000, 100_000])
def test_fp64_forces_of_unwrapped_positions(k):
    n = 1728
    r = np.random.default_rng(7)
    g = np.stack(np.meshgrid(*[np.arange(12)] * 3, indexing="ij")).reshape(3, -1)
    pos = np.ascontiguousarray((g + 0.5 + r.uniform(-0.08, 0.08, g.shape)) * (L / 12))
    atoms = amber.AtomData(np.full(n, 3.0), np.full(n, 0.1), np.full(n, 12.0), r.uniform(-0.3, 0.3, n),
                           np.full(n, 1, np.uint8), np.zeros(n, np.uint32), [])
    p = backend.SimParams(box_size=(L,) * 3, periodic=True, r_cutoff=10.0, r_skin=12.0, r_switch=8.0, coulomb=True,
                          precision=backend.PRECISION_FP64)
    be = backend.CudaBackend(atoms, amber.BondedTopology.empty(), p)
    be.build_neighbor_list(pos)
    f0, e0 = be.compute_forces(pos).copy(), be.potential_energy()
    far = np.ascontiguousarray(pos + L * k * r.integers(-1, 2, (3, n)))
    f, e = be.compute_forces(far).copy(), be.potential_energy()
    be.close()
    assert np.max(np.abs(f - f0)) <= 6.2e-11 * k + 1e-9
    # half of n * 100 neighbours inside the cutoff, the same bound of a length times |F| <= 1 each
    assert abs(e - e0) <= 100 * n * 2.1e-14 * k + 1e-9 * abs(e0)
