"""Forests whose levels interleave in the caller's block order: fields,
populations and equilibrium states travel as one array in that order, each
level's kernel placing its blocks.  The populations read back after setting
them are the collided ones block by block (single-block contexts collide the
same block alone), and the fields those of the populations."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ob():
    return pytest.importorskip("octlb_b200")


@pytest.mark.parametrize("prec", ["fp32", "fp16"])
def test_interleaved_levels_keep_block_order(ob, prec):
    from octlb_b200 import cases
    mesh, _, info = cases.cavity_forest(cells=32, n=8, lid=0.1, tau=0.6, band_cells=8)
    assert np.any(np.diff(mesh.levels) != 0) and len(set(mesh.levels.tolist())) == 2
    p = ob.FP16_SHIFTED if prec == "fp16" else ob.FP32
    rng = np.random.default_rng(2)
    pops = 1e-3 * rng.standard_normal((mesh.n_blocks, 8, 8, 8, 19))
    lat = ob.GpuLattice(mesh, info["omega"], precision=p)
    lat.set_populations(pops)
    g = lat.get_populations()
    rho, u = lat.get_fields()
    one = ob.Mesh(8, [0], [0, 0, 0, 1, 1, 1], tree_boundary=[(0, d) for d in range(6)],
                  tree_boundary_spec=[[ob.TB_WALL, 0, 0, 0, -1, 0, 0, 0]] * 6)
    ref = ob.GpuLattice(one, info["omega"], precision=p)
    for b in (0, 1, mesh.n_blocks // 2, mesh.n_blocks - 1):
        ref.set_populations(pops[b:b + 1])
        assert np.array_equal(ref.get_populations()[0], g[b])
        r1, u1 = ref.get_fields()
        assert np.array_equal(r1[0], rho[b]) and np.array_equal(u1[0], u[b])
    rho0, u0 = 1.0 + 0.01 * rng.standard_normal(rho.shape), 0.02 * rng.standard_normal(u.shape)
    lat.set_equilibrium(rho0.reshape(-1), u0.reshape(-1, 3))
    g = lat.get_populations()
    for b in (0, mesh.n_blocks - 1):
        ref.set_equilibrium(rho0[b].reshape(-1), u0[b].reshape(-1, 3))
        assert np.array_equal(ref.get_populations()[0], g[b])
    ref.close()
    lat.close()
