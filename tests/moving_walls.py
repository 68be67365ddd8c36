"""Meshes whose walls move on one face, any way: shared by the tests of the
slot-map step's row tables (test_map_rows.py, test_gpu_map_walls.py)."""
import numpy as np

FACES, AXES = range(6), range(3)
NAMES = ([f"face{d}_u{a}_{n}" for n in (8, 16) for d in FACES for a in AXES] +
         ["duct_uniform", "duct_parabola_y", "duct_parabola_z", "duct_16", "cylinder_closed_z", "cylinder_closed_z_16"])


def _walls(ob, forest, n, moving, outflow=None):
    """Tree-boundary walls at rest except `moving` = {direction: (u, profile
    axis, lo, hi)}, and an outflow on direction `outflow`."""
    spec = np.zeros((len(forest.tree_boundary), 8))
    spec[:, 0], spec[:, 4] = ob.TB_WALL, -1
    for k, (_, d) in enumerate(forest.tree_boundary):
        if int(d) == outflow:
            spec[k, 0] = ob.TB_OUTFLOW
        elif int(d) in moving:
            u, axis, lo, hi = moving[int(d)]
            spec[k, 1:7] = [*u, axis, lo, hi]
    return ob.Mesh.from_forest(forest, n, tree_boundary_spec=spec)


def mesh(ob, name):
    """(mesh, options) of one of NAMES."""
    from octlb_b200 import cases
    if name.startswith("face"):  # one closed block, one wall moving along one axis
        d, a, n = int(name[4]), int(name[7]), int(name.split("_")[2])
        f = ob.Forest((1, 1, 1), (0, 0, 0), (0, 0, 0, 1, 1, 1)).balance().build()
        u = np.zeros(3)
        u[a] = 0.05
        return _walls(ob, f, n, {d: (u, -1, 0.0, 0.0)}), {}
    if name.startswith("duct"):  # inlet -x, outflow +x, walls at rest in y and z
        n = 16 if name == "duct_16" else 8
        f = ob.Forest((3, 2, 2), (0, 0, 0), (0, 0, 0, 3, 2, 2)).balance().build()
        axis = {"duct_parabola_y": 1, "duct_parabola_z": 2}.get(name, -1)
        return _walls(ob, f, n, {0: ([0.05, 0.0, 0.0], axis, 0.0, 2.0)}, outflow=1), {}
    n = 16 if name.endswith("_16") else 8
    h = 64 if n == 16 else 32
    m, _, _ = cases.cylinder_forest(length=128, height=h, n=n, diameter=8.0, center=(32.0, h / 2), levels=2,
                                    u_max=0.05, re=40.0, periodic_z=False)
    return m, dict(stream_mode=ob.STREAM_LINKS, drag=True)
