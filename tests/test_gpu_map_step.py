"""The slot-map step (z pairs of cells per thread, packed collide, the default
on forest levels of 8^3 and 16^3 blocks) against the plain one-cell step: same
pulls, same arithmetic, so populations and forces are bitwise equal -- on
random states, with walls, moving walls, outflow copies, open halos, coupler
saves, Bouzidi links, solid and non-kBulk cells beside kBulk ones in a pair,
and FP16 scales that are and are not powers of two (the latter with walls at
rest: there the wall term and the conversion of the value it is added to may
or may not contract into one rounding, kernel by kernel).  Under ConstRhoBGK the
two sum the statistics in different orders (FP64, cells summed in pairs in
FP32 first): the average may differ in its last FP32 digits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ob():
    return pytest.importorskip("octlb_b200")


def random_state(mesh, seed=3):
    rng = np.random.default_rng(seed)
    return 1e-3 * rng.standard_normal((mesh.n_blocks, mesh.n, mesh.n, mesh.n, 19))


def meshes(ob, name, wall=1.0):
    from octlb_b200 import cases
    if name == "one_block":
        return cases.cavity_forest(cells=8, n=8, lid=0.1 * wall, tau=0.6), {}
    if name == "one_block_16":
        return cases.cavity_forest(cells=16, n=16, lid=0.1 * wall, tau=0.6), {}
    if name == "cavity_band":
        return cases.cavity_forest(cells=32, n=8, lid=0.1 * wall, tau=0.6, band_cells=8), {}
    if name == "cavity_kinds":  # scattered non-kBulk cells: pairs with one of each
        mesh, init, info = cases.cavity_forest(cells=32, n=8, lid=0.1 * wall, tau=0.6)
        rng = np.random.default_rng(5)
        mesh.kinds[rng.random(mesh.kinds.shape) < 0.2] = ob.BOUNCE_BACK
        return (mesh, init, info), {}
    links = dict(stream_mode=ob.STREAM_LINKS, drag=True)
    if name == "cylinder":
        return cases.cylinder_forest(length=128, height=32, n=8, diameter=8.0, center=(32.0, 16.0), levels=2,
                                     u_max=0.05 * wall, re=40.0), links
    return cases.cylinder_forest(length=128, height=64, n=16, diameter=8.0, center=(32.0, 32.0), levels=2,
                                 u_max=0.05 * wall, re=40.0), links


def run(ob, monkeypatch, variant, name, precision, steps, scale=None, const_rho=False):
    (mesh, _, info), kw = meshes(ob, name, wall=0.0 if scale == 50000.0 else 1.0)
    omega = 1.0 / 0.6
    monkeypatch.setenv("OCTLB_STEP_KERNEL", variant)
    lat = ob.GpuLattice(mesh, omega, precision=precision, init_pops=random_state(mesh), fp16_scale=scale, **kw)
    if const_rho:
        lat.set_const_rho(True)
    lat.advance(steps)
    out = lat.get_populations(), lat.force() if kw else np.zeros(3), lat.average_rho()
    lat.close()
    return out


@pytest.mark.parametrize("prec,scale", [("fp32", None), ("fp16", None), ("fp16", 32768.0), ("fp16", 50000.0)])
@pytest.mark.parametrize("name,steps", [("one_block", 5), ("one_block_16", 3), ("cavity_band", 3), ("cavity_kinds", 3),
                                        ("cylinder", 4), ("cylinder_16", 2)])
def test_map_step_bitwise_equals_plain(ob, name, steps, prec, scale, monkeypatch):
    p = ob.FP16_SHIFTED if prec == "fp16" else ob.FP32
    a = run(ob, monkeypatch, "map", name, p, steps, scale)
    b = run(ob, monkeypatch, "plain", name, p, steps, scale)
    assert np.all(np.isfinite(a[0]))
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])


@pytest.mark.parametrize("prec", ["fp32", "fp16"])
@pytest.mark.parametrize("n,links", [(8, False), (16, False), (8, True)])
def test_map_step_const_rho(ob, n, links, prec, monkeypatch):
    """ConstRhoBGK on a closed box of level-0 blocks (an advance_one is one
    step), walls at rest, with scattered solid cells under the links rule.  The
    first step collides at the average the initial state gave, the same in both
    kernels: bitwise equal populations.  The second step's average comes from
    the first step's statistics: streaming in the closed box keeps the sum of
    the kBulk cells' populations, so it is 1 + mean(sum g0) + (1 - avg1); a
    cell's density is a 19-term FP32 sum (error <= 19 * 2^-24 * sum |f| < 2e-8
    for sum |f| < 0.02)."""
    f = ob.Forest((4, 3, 2), (0, 0, 0), (0, 0, 0, 4, 3, 2)).balance().build()
    spec = np.zeros((len(f.tree_boundary), 8))
    spec[:, 0], spec[:, 4] = ob.TB_WALL, -1
    mesh = ob.Mesh.from_forest(f, n, tree_boundary_spec=spec)
    if links:
        rng = np.random.default_rng(11)
        mesh.kinds[:, 2:-2, 2:-2, 2:-2][rng.random((mesh.n_blocks, n - 4, n - 4, n - 4)) < 0.2] = ob.SOLID
    kw = dict(stream_mode=ob.STREAM_LINKS) if links else {}
    p = ob.FP16_SHIFTED if prec == "fp16" else ob.FP32
    res = []
    for variant in ("map", "plain"):
        monkeypatch.setenv("OCTLB_STEP_KERNEL", variant)
        lat = ob.GpuLattice(mesh, 1.0 / 0.6, precision=p, init_pops=random_state(mesh), **kw)
        lat.set_const_rho(True)
        g0 = lat.get_populations()
        lat.advance(1)
        g1, avg1 = lat.get_populations(), lat.average_rho()
        lat.advance(1)
        res.append((g1, avg1, lat.average_rho()))
        lat.close()
    assert np.array_equal(res[0][0], res[1][0]) and res[0][1] == res[1][1]
    bulk = mesh.kinds == ob.BULK
    want = 1.0 + g0[bulk].sum(axis=-1).mean() + 1.0 - avg1
    assert abs(res[0][2] - want) <= 2e-8 and abs(res[1][2] - want) <= 2e-8
