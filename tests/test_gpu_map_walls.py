"""Moving walls on every face and along every axis: the slot-map step against
the plain one-cell step, bitwise (same pulls, same arithmetic), on random
states.  The first moving position of a level may lie at the start of a z row
(a lid along z, an inlet between z walls at rest), in the row before it or in
neither: the step's row path numbers the wall terms along the row."""
import numpy as np
import pytest

from moving_walls import NAMES, mesh

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ob():
    return pytest.importorskip("octlb_b200")


def run(ob, monkeypatch, variant, name, precision, mode):
    m, kw = mesh(ob, name)
    monkeypatch.setenv("OCTLB_STEP_KERNEL", variant)
    init = 1e-3 * np.random.default_rng(4).standard_normal((m.n_blocks, m.n, m.n, m.n, 19))
    lat = ob.GpuLattice(m, 1.0 / 0.6, precision=precision, init_pops=init, **kw)
    if mode == "const_rho":
        lat.set_const_rho(True)
    lat.advance(1 if mode == "const_rho" else 3)
    out = lat.get_populations(), lat.force() if kw else np.zeros(3)
    lat.close()
    return out


@pytest.mark.parametrize("prec", ["fp32", "fp16"])
@pytest.mark.parametrize("name", NAMES)
def test_moving_walls_bitwise_equal_plain(ob, name, prec, monkeypatch):
    p = ob.FP16_SHIFTED if prec == "fp16" else ob.FP32
    a = run(ob, monkeypatch, "map", name, p, "bgk")
    b = run(ob, monkeypatch, "plain", name, p, "bgk")
    assert np.all(np.isfinite(a[0]))
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])


@pytest.mark.parametrize("prec", ["fp32", "fp16"])
@pytest.mark.parametrize("name", ["face3_u2_8", "face3_u2_16", "face0_u0_8", "duct_uniform"])
def test_moving_walls_const_rho(ob, name, prec, monkeypatch):
    """One level, one step: both kernels collide at the average of the initial
    state."""
    p = ob.FP16_SHIFTED if prec == "fp16" else ob.FP32
    a = run(ob, monkeypatch, "map", name, p, "const_rho")
    b = run(ob, monkeypatch, "plain", name, p, "const_rho")
    assert np.array_equal(a[0], b[0])
