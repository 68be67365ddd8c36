"""Long advances put sixteen advance_one calls in a CUDA graph where a call is a
few short launches: the same states, forces, statistics and counters as one call
at a time, from either buffer parity, with the drag's side stream, body forces,
two levels, ConstRhoBGK and the one-buffer order."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ob():
    return pytest.importorskip("octlb_b200")


def walls(ob, forest, n):
    spec = np.zeros((len(forest.tree_boundary), 8))
    spec[:, 0], spec[:, 4] = ob.TB_WALL, -1
    spec[forest.tree_boundary[:, 1] == 3, 1] = 0.05
    return ob.Mesh.from_forest(forest, n, tree_boundary_spec=spec)


def make(ob, name, precision):
    kw = {}
    if name in ("box", "box_aa"):
        mesh = ob.Mesh(32, [0], [0, 0, 0, 1, 1, 1], periodic=1)
        if name == "box_aa":
            kw["stream_order"] = ob.ORDER_AA
    elif name.startswith("two_levels"):
        mesh = walls(ob, ob.Forest((2, 2, 2), (0, 0, 0), (0, 0, 0, 2, 2, 2)).refine_box((0, 1.2, 0, 2, 2, 2), 1).balance().build(), 8)
    else:
        mesh = walls(ob, ob.Forest((4, 2, 2), (0, 0, 0), (0, 0, 0, 4, 2, 2)).balance().build(), 8)
    if name == "drag":
        mesh.kinds[5, 2:6, 2:6, 2:6] = ob.SOLID
        mesh.obstacle = (mesh.kinds == ob.SOLID).astype(np.uint8)
        kw.update(stream_mode=ob.STREAM_LINKS, drag=True)
    rng = np.random.default_rng(3)
    shape = (mesh.n_blocks, mesh.n, mesh.n, mesh.n)
    lat = ob.GpuLattice(mesh, 1.0 / 0.6, precision=precision, **kw)
    if name.endswith("const_rho"):
        lat.set_const_rho(True)
    lat.set_equilibrium((1.0 + 0.01 * rng.standard_normal(shape)).reshape(-1), (0.02 * rng.standard_normal(shape + (3,))).reshape(-1, 3))
    if name == "force":
        lat.set_body_force(1e-5 * rng.standard_normal((mesh.n_blocks, mesh.n ** 3, 3)))
    return lat, "drag" in kw


@pytest.mark.parametrize("prec", ["fp32", "fp16"])
@pytest.mark.parametrize("name", ["box", "box_aa", "level", "level_const_rho", "force", "drag", "two_levels", "two_levels_const_rho"])
def test_long_advances_equal_single_calls(ob, name, prec):
    res = []
    for chunks in ((32, 1, 50, 7), (1,) * 90):
        lat, drag = make(ob, name, ob.FP16_SHIFTED if prec == "fp16" else ob.FP32)
        for n in chunks:
            lat.advance(n)
        out = [lat.get_populations(), *lat.get_fields(), np.array(lat.average_rho()), np.array(lat.counters())]
        if drag:
            total, steps = lat.force_sum()
            out += [lat.force(), total, np.array(steps)]
        res.append(out)
        lat.close()
    for a, b in zip(*res):
        assert np.all(np.isfinite(a)) and np.array_equal(a, b)
