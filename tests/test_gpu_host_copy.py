"""Large pageable arrays go through pinned buffers by several threads, pinned
ones directly: the same bytes either way, at sizes around the threshold (8 MB), from several
contexts at once."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ob():
    return pytest.importorskip("octlb_b200")


@pytest.mark.parametrize("n", [38, 40, 65])  # populations 8.34 MB (below 8 MiB), 9.7 and 41.7 MB
def test_pageable_and_pinned_arrays(ob, n):
    import torch
    rng = np.random.default_rng(n)
    pops = 1e-3 * rng.standard_normal((n ** 3, 19))
    mesh = ob.Mesh(n, [0], [0, 0, 0, 1, 1, 1], periodic=1)
    lat = ob.GpuLattice(mesh, 1.0 / 0.6)
    pinned = torch.empty(pops.size, dtype=torch.float64, pin_memory=True)
    pinned.numpy()[:] = pops.reshape(-1)
    lat.set_populations(pops)
    a = lat.get_populations()
    ra, ua = lat.get_fields()
    lat.set_populations(pinned.numpy())
    b = lat.get_populations()
    rp = torch.empty(n ** 3, dtype=torch.float64, pin_memory=True).numpy()
    up = torch.empty((n ** 3, 3), dtype=torch.float64, pin_memory=True).numpy()
    lat.get_fields(rp, up)
    assert np.array_equal(a, b)
    assert np.array_equal(ra.reshape(-1), rp) and np.array_equal(ua.reshape(-1), up.reshape(-1))
    rho = 1.0 + 0.01 * rng.standard_normal(n ** 3)
    u = 0.02 * rng.standard_normal((n ** 3, 3))
    lat.set_equilibrium(rho, u)
    a = lat.get_populations()
    rp[:], up[:] = rho, u
    lat.set_equilibrium(rp, up)
    assert np.array_equal(a, lat.get_populations())
    lat.close()


def test_two_contexts_at_once(ob):
    n = 56
    out = [None, None]

    def work(k):
        rng = np.random.default_rng(k)
        pops = 1e-3 * rng.standard_normal((n ** 3, 19))
        lat = ob.GpuLattice(ob.Mesh(n, [0], [0, 0, 0, 1, 1, 1], periodic=1), 1.0)  # omega = 1: the equilibrium
        for _ in range(3):
            lat.set_populations(pops)
            g = lat.get_populations()
        rho, _ = lat.get_fields()
        out[k] = np.max(np.abs(rho.reshape(-1) - (1.0 + pops.sum(axis=1)))), np.max(np.abs(g.sum(axis=-1).reshape(-1) - pops.sum(axis=1)))
        lat.close()

    ts = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    [t.start() for t in ts]
    [t.join() for t in ts]
    # FP32 storage of populations below 0.01: 19 roundings of 2^-24 * 0.04
    assert all(max(o) < 19 * 2.0 ** -24 * 0.04 * 4 for o in out)
