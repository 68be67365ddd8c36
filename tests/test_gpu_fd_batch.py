"""Steps of one graph skip the finite-difference pass's store and count the
boundary clock from the graph's start: the same populations, fields and
average as stepping one call at a time, with an inlet ramp that depends on the
clock, ConstRhoBGK on and off."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ob():
    return pytest.importorskip("octlb_b200")


@pytest.mark.parametrize("prec", ["fp32", "fp16"])
@pytest.mark.parametrize("n,const_rho", [(9, True), (16, False)])
def test_batched_steps_equal_single_steps(ob, n, const_rho, prec):
    from octlb_b200 import cases
    mesh, init, _ = cases.cavity_forest(cells=n, n=n, lid=0.0, tau=0.7)
    types = [ob.FD_VELOCITY, ob.FD_PRESSURE, ob.FD_VELOCITY, ob.FD_VELOCITY, ob.FD_VELOCITY, ob.FD_VELOCITY]
    u_wall = np.zeros((6, 3))
    u_wall[3, 0] = 0.02
    inlet = np.zeros((6, 3))
    inlet[0, 0] = 0.03
    res = []
    for calls in ([50, 33, 1, 6], [1] * 90):  # 2 graphs of 16, then singles; 2 graphs; singles
        lat = ob.GpuLattice(ob.stamp_fd_kinds(mesh, types), 1.0 / 0.7,
                            precision=ob.FP16_SHIFTED if prec == "fp16" else ob.FP32, init_pops=init)
        if const_rho:
            lat.set_const_rho(True)
        lat.set_fd_boundary(types, u_wall, inlet_u=inlet, ramp_end_t=60.0)
        for c in calls:
            lat.advance(c)
        res.append((lat.get_populations(), *lat.get_fields(), lat.average_rho(), lat.counters()))
        lat.close()
    a, b = res
    assert np.all(np.isfinite(a[0])) and np.max(np.abs(a[2])) > 1e-3
    assert all(np.array_equal(x, y) for x, y in zip(a[:3], b[:3]))
    assert a[3] == b[3] and a[4] == b[4]
