"""Host arrays of every size are read and written in the order of the stream
that the context was given, also where that is a thread's default stream (a
handle that names another stream in another thread)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PER_THREAD = 2  # cudaStreamPerThread


@pytest.fixture(scope="module")
def ob():
    return pytest.importorskip("octlb_b200")


def outputs(ob, mesh, init, stream, steps):
    lat = ob.GpuLattice(mesh, 1.0 / 0.6)
    if stream:
        lat.set_stream(stream)
    lat.set_populations(init)
    got = []
    for _ in range(3):  # the copies follow queued steps
        lat.advance(steps)
        got.append(lat.get_populations())
        lat.advance(steps)
        got.extend(lat.get_fields())
    lat.close()
    return got


@pytest.mark.parametrize("n", [24, 96])  # below and above the staged copies' size
def test_per_thread_default_stream(ob, n):
    mesh = ob.Mesh(n, [0], [0, 0, 0, 1, 1, 1], periodic=1)
    init = 1e-3 * np.random.default_rng(n).standard_normal((n ** 3, 19))
    want = outputs(ob, mesh, init, None, 200)
    for a, b in zip(want, outputs(ob, mesh, init, PER_THREAD, 200)):
        assert np.array_equal(a, b)
