"""A context's large pageable arrays take the driver's path until the pinned
buffers would have repaid their making, then those: the same bytes before, at and
after the change, in a context alone and beside one that has the buffers."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ob():
    return pytest.importorskip("octlb_b200")


@pytest.mark.parametrize("beside", [False, True])
@pytest.mark.parametrize("n", [40, 64])  # populations of 9.7 and 39.8 MB: the third and first copy back change the path
def test_same_bytes_on_both_paths(ob, n, beside):
    rng = np.random.default_rng(n)
    mesh = ob.Mesh(n, [0], [0, 0, 0, 1, 1, 1], periodic=1)
    other = None
    if beside:
        other = ob.GpuLattice(ob.Mesh(72, [0], [0, 0, 0, 1, 1, 1], periodic=1), 1.0 / 0.6)
        other.get_populations()  # 56.7 MB: the buffers are made
    lat = ob.GpuLattice(mesh, 1.0 / 0.6)
    small = ob.GpuLattice(mesh, 1.0 / 0.6)  # a second context, on the driver's path throughout
    for k in range(7):
        pops = 1e-3 * rng.standard_normal((n ** 3, 19))
        lat.set_populations(pops)
        small.set_equilibrium(1.0 + pops.sum(axis=1), pops[:, :3].copy())
        a = lat.get_populations()
        lat.set_populations(pops)
        assert np.array_equal(a, lat.get_populations())
        rho, u = small.get_fields()
        assert np.allclose(rho.reshape(-1), 1.0 + pops.sum(axis=1), rtol=0, atol=19 * 2.0 ** -23)
    for l in (lat, small, other):
        if l is not None:
            l.close()
