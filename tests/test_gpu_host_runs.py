"""Forests move in and out in runs of blocks of the caller's order.  A mesh
whose blocks are listed level by level needs no reordering; the same mesh in
the forest's interleaved order must give the same states, fields and ConstRhoBGK
averages, block for block and bit for bit.  The staging a context keeps is what
its largest level takes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ob():
    return pytest.importorskip("octlb_b200")


def by_level(ob, m):
    """The mesh with its blocks sorted by level, and where each came from."""
    order = np.argsort(m.levels, kind="stable")
    new = np.empty_like(order)
    new[order] = np.arange(len(order))
    same, cf, tb, links = m.same_level.copy(), m.coarse_fine.copy(), m.tree_boundary.copy(), m.link_cells.copy()
    same[:, [0, 2]] = new[same[:, [0, 2]]]
    cf[:, :5] = new[cf[:, :5]]
    tb[:, 0] = new[tb[:, 0]]
    links[:, 0] = new[links[:, 0]]
    s = ob.Mesh(m.n, m.levels[order], m.bounds[order], kinds=m.kinds[order], same_level=same, coarse_fine=cf,
                coarse_fine_bounds=m.coarse_fine_bounds, tree_boundary=tb, tree_boundary_spec=m.tree_boundary_spec,
                link_cells=links, link_q=m.link_q, obstacle=None if m.obstacle is None else m.obstacle[order])
    return s, order


def mesh_of(ob, name):
    from octlb_b200 import cases
    if name == "cylinder":  # three levels
        return cases.cylinder_forest(length=128, height=64, n=8, diameter=8.0, center=(40.0, 32.0), levels=3)[0], dict(
            stream_mode=ob.STREAM_LINKS, drag=True)
    cells, n, band = {"cavity": (32, 8, 8), "cavity_4": (16, 4, 4), "cavity_16": (64, 16, 16)}[name]
    return cases.cavity_forest(cells=cells, n=n, lid=0.1, band_cells=band)[0], {}


@pytest.mark.parametrize("prec", ["fp32", "fp16"])
@pytest.mark.parametrize("name,const_rho", [("cavity", False), ("cavity", True), ("cavity_4", False), ("cavity_4", True),
                                            ("cavity_16", True), ("cylinder", False)])
def test_interleaved_order_equals_level_order(ob, name, const_rho, prec):
    mesh, kw = mesh_of(ob, name)
    sorted_mesh, order = by_level(ob, mesh)
    assert not np.array_equal(order, np.arange(len(order)))
    rng = np.random.default_rng(7)
    shape = (mesh.n_blocks, mesh.n, mesh.n, mesh.n)
    pops = 1e-3 * rng.standard_normal(shape + (19,))
    rho, u = 1.0 + 0.01 * rng.standard_normal(shape), 0.02 * rng.standard_normal(shape + (3,))
    res = []
    for m, pick in ((mesh, np.arange(mesh.n_blocks)), (sorted_mesh, order)):
        lat = ob.GpuLattice(m, 1.0 / 0.6, precision=ob.FP16_SHIFTED if prec == "fp16" else ob.FP32, **kw)
        if const_rho:
            lat.set_const_rho(True)
        out = []
        for start in (lambda: lat.set_populations(pops[pick]),
                      lambda: lat.set_equilibrium(rho[pick].reshape(-1), u[pick].reshape(-1, 3))):
            start()
            out.append(lat.get_populations())
            lat.advance(2)
            out += [lat.get_populations(), *lat.get_fields()]
            out.append(np.full(mesh.n_blocks, lat.average_rho()))
        res.append([np.asarray(a).reshape((mesh.n_blocks, -1)) for a in out])
        lat.close()
    for a, b in zip(*res):
        assert np.all(np.isfinite(a)) and np.array_equal(a[order], b)


@pytest.mark.parametrize("const_rho", [False, True])
def test_interleaved_order_with_fd_walls(ob, const_rho):
    """The rewritten boundary cells' fields land in their blocks' places too."""
    f = ob.Forest((1, 1, 1), (0, 0, 0), (0, 0, 0, 1, 1, 1)).refine_uniform(2)
    f.refine_box((0.26, 0.26, 0.26, 0.74, 0.74, 0.74), 3).balance().build()
    mesh = ob.Mesh.from_forest(f, 8)
    types = [ob.FD_VELOCITY] * 6
    u_wall = np.zeros((6, 3))
    u_wall[3, 0] = 0.03
    mesh = ob.stamp_fd_kinds(mesh, types)
    sorted_mesh, order = by_level(ob, mesh)
    assert not np.array_equal(order, np.arange(len(order)))
    rng = np.random.default_rng(8)
    shape = (mesh.n_blocks, 8, 8, 8)
    rho, u = 1.0 + 0.01 * rng.standard_normal(shape), 0.02 * rng.standard_normal(shape + (3,))
    res = []
    for m, pick in ((mesh, np.arange(mesh.n_blocks)), (sorted_mesh, order)):
        lat = ob.GpuLattice(m, 1.0 / 0.6)
        if const_rho:
            lat.set_const_rho(True)
        lat.set_equilibrium(rho[pick].reshape(-1), u[pick].reshape(-1, 3))
        lat.set_fd_boundary(types, u_wall)
        out = []
        for _ in range(2):
            lat.advance(3)
            out += [lat.get_populations(), *lat.get_fields()]
        res.append([np.asarray(a).reshape((mesh.n_blocks, -1)) for a in out])
        lat.close()
    for a, b in zip(*res):
        assert np.all(np.isfinite(a)) and np.array_equal(a[order], b)


def test_staging_held_is_the_largest_level(ob):
    import torch
    from octlb_b200 import cases
    mesh = cases.cavity_forest(cells=64, n=8, lid=0.1, band_cells=8)[0]
    lat = ob.GpuLattice(mesh, 1.0 / 0.6)
    lat.advance(1)
    lat.synchronize()
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    lat.get_fields()
    pops = lat.get_populations()
    lat.set_populations(pops)
    held = free - torch.cuda.mem_get_info()[0]
    cells = max(np.bincount(mesh.levels)) * mesh.n ** 3
    # rho, u and populations of the largest level in FP64, and a 2 MB granule
    # for each buffer (both arrays, block ids of two levels)
    assert held <= cells * (19 + 3) * 8 + 4 * 2 ** 21, (held, cells)
    lat.close()
