"""The row tables of the slot-map step against the slot maps they stand for:
the planning pass replays, for every pair of cells and direction of every
block with uniform rows, the position and the moving-wall marker that the
step's row path forms, and refuses a mesh where they differ."""
import pytest

from moving_walls import NAMES, mesh


@pytest.mark.parametrize("name", NAMES)
def test_row_tables_match_the_slot_maps(ob, name):
    m, kw = mesh(ob, name)
    levels = ob.plan(m, 1.0 / 0.6, **kw)
    assert sum(l["blocks"] for l in levels) == m.n_blocks


@pytest.mark.parametrize("cells,n,band", [(16, 16, 0), (32, 8, 8), (64, 16, 0)])
def test_row_tables_of_cavities(ob, cells, n, band):
    from octlb_b200 import cases
    m, _, info = cases.cavity_forest(cells=cells, n=n, lid=0.1, band_cells=band)
    ob.plan(m, info["omega"])
