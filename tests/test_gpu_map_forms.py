"""The slot-map step's two launch forms on either side of the CTA counts where
the choice between them falls (148 SMs: 740 CTAs of 256 cells, 296 of 512 under
ConstRhoBGK), bitwise against the plain step."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ob():
    return pytest.importorskip("octlb_b200")


@pytest.mark.parametrize("prec", ["fp32", "fp16"])
@pytest.mark.parametrize("bricks,const_rho", [((8, 37, 1), True), ((9, 11, 3), True), ((37, 10, 1), False), ((53, 7, 1), False)])
def test_forms_bitwise_equal_plain(ob, bricks, const_rho, prec, monkeypatch):
    f = ob.Forest(bricks, (0, 0, 0), (0, 0, 0, *bricks)).balance().build()
    spec = np.zeros((len(f.tree_boundary), 8))
    spec[:, 0], spec[:, 4] = ob.TB_WALL, -1
    spec[f.tree_boundary[:, 1] == 3, 3] = 0.05
    mesh = ob.Mesh.from_forest(f, 8, tree_boundary_spec=spec)
    init = 1e-3 * np.random.default_rng(9).standard_normal((mesh.n_blocks, 8, 8, 8, 19))
    res = []
    for variant in ("map", "plain"):
        monkeypatch.setenv("OCTLB_STEP_KERNEL", variant)
        lat = ob.GpuLattice(mesh, 1.0 / 0.6, precision=ob.FP16_SHIFTED if prec == "fp16" else ob.FP32, init_pops=init)
        lat.set_const_rho(const_rho)
        lat.advance(1 if const_rho else 2)  # ConstRhoBGK: the initial state's average in both
        res.append(lat.get_populations())
        lat.close()
    assert np.all(np.isfinite(res[0])) and np.array_equal(*res)
