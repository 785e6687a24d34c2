"""Strokes of a solid material through water, whose columns run side by side, against the oracle's cell after
cell: spheres around every limit of that path (list length, chunk of 4096, columns that fit, water that has to
go to the sides, films of hidden water, lists that go down a column or name a voxel twice)."""
import numpy as np
import pytest

from conftest import assert_same_digest, oracle_for

pytestmark = pytest.mark.gpu
STONE, WATER = 3, 5


def pool(vf, orc, ny=64, top=40, lid=None):
    w = vf.World(48, ny, 48)
    w.fill_box(0, 0, 0, 47, 3, 47, STONE)
    for b in ((0, 0, 47, 1), (0, 46, 47, 47), (0, 0, 1, 47), (46, 0, 47, 47)):
        w.fill_box(b[0], 4, b[1], b[2], ny - 1, b[3], STONE)
    w.fill_box(2, 4, 2, 45, top, 45, WATER)
    if lid is not None:
        w.fill_box(20, lid, 20, 27, lid, 27, STONE)
    return vf.FluidSim(w, device=0), oracle_for(orc, w)


def sphere(c, r):
    a = np.arange(-r, r + 1)
    z, y, x = np.meshgrid(a, a, a, indexing="ij")
    keep = x * x + y * y + z * z <= r * r
    return np.stack([x[keep] + c[0], y[keep] + c[1], z[keep] + c[2]], 1).astype(np.int32)


def same(sim, o, ticks=0):
    assert_same_digest(sim, o)
    assert sim.partial_count() == o.partial_count()
    if ticks:
        sim.tick(ticks)
        o.tick(ticks)
        assert_same_digest(sim, o)


@pytest.mark.parametrize("r", [1, 2, 3, 6, 10])  # 7, 33, 123, 925 and 4169 cells
@pytest.mark.parametrize("at", [(24, 16, 24), (24, 38, 24), (3, 30, 5), (24, 60, 24)])  # deep, at the surface, in a wall, past the top
def test_spheres(vf, orc, r, at):
    sim, o = pool(vf, orc)
    cells = sphere(at, r)
    assert sim.apply_brush(cells, STONE) == o.apply_brush(cells, STONE)
    same(sim, o)
    cells = sphere((at[0] + r, at[1] + 1, at[2]), r)  # a second stroke beside it: partly stone, raised surface
    assert sim.apply_brush(cells, STONE) == o.apply_brush(cells, STONE)
    same(sim, o, 3)
    cells = sphere((at[0] - 1, at[1] + 2, at[2] + r), r)  # in water that has moved: partial and hidden volumes
    assert sim.apply_brush(cells, STONE) == o.apply_brush(cells, STONE)
    same(sim, o, 2)
    sim.close()


@pytest.mark.parametrize("lid", [19, 24, 41])  # in the stroke, just above it, on the surface: water goes to the sides
def test_water_that_does_not_fit_its_column(vf, orc, lid):
    sim, o = pool(vf, orc, lid=lid)
    cells = sphere((24, 16, 24), 6)
    assert sim.apply_brush(cells, STONE) == o.apply_brush(cells, STONE)
    same(sim, o, 2)
    sim.close()


@pytest.mark.parametrize("ny,top", [(64, 40), (160, 150)])  # the tall one: more than 128 cells of column above
@pytest.mark.parametrize("order", ["down", "twice", "shuffled", "outside"])
def test_lists(vf, orc, ny, top, order):
    sim, o = pool(vf, orc, ny, top)
    cells = sphere((24, 16, 24), 4)
    if order == "down":
        cells = cells[::-1]
    elif order == "twice":
        cells = np.concatenate([cells, cells[:40]])
    elif order == "shuffled":
        cells = np.random.default_rng(3).permutation(cells)
    else:
        cells = np.concatenate([cells, np.array([[-5, 16, 24], [24, -1, 24], [24, ny, 24], [500, 16, 24]], np.int32)])
    cells = np.ascontiguousarray(cells)
    assert sim.apply_brush(cells, STONE) == o.apply_brush(cells, STONE)
    same(sim, o, 2)
    sim.close()


def test_water_with_nowhere_to_go(vf, orc):
    """A closed tank full of water: a displaced cell's water finds no room above or beside it and is gone, in
    columns that touch each other."""
    w = vf.World(40, 40, 40)
    w.fill_box(0, 0, 0, 39, 39, 39, STONE)
    w.fill_box(4, 4, 4, 35, 35, 35, WATER)
    sim, o = vf.FluidSim(w, device=0), oracle_for(orc, w)
    for c, r in (((20, 20, 20), 6), ((24, 22, 20), 5), ((6, 30, 6), 9)):
        cells = sphere(c, r)
        assert sim.apply_brush(cells, STONE) == o.apply_brush(cells, STONE)
        same(sim, o)
    same(sim, o, 2)
    sim.close()


# lists in no order: what a chunk leaves for later may lie between cells of its column that it takes
@pytest.mark.parametrize("order", [0, 1, 2, 4, 5, "low high twice middle", "stairs", "zigzag", "far up"])
def test_lists_in_no_order(vf, orc, order):
    sim, o = pool(vf, orc, *((160, 150) if order == "far up" else ()))
    cells = sphere((24, 16, 24), 4)
    if isinstance(order, int):
        cells = np.random.default_rng(order).permutation(cells)
    elif order == "low high twice middle":
        cells = np.array([[5, 5, 5], [5, 7, 5], [5, 5, 5], [5, 6, 5]] + [[10 + i, 6, 9] for i in range(12)], np.int32)
    elif order == "stairs":  # every column: the lowest cell, the highest, then the ones between downwards
        cells = np.array([[x, y, 20] for x in range(10, 20) for y in (5, 12, 11, 10, 9, 8, 7, 6)], np.int32)
    elif order == "zigzag":  # layers in turn over all columns, each column up and down
        cells = np.array([[x, y, 20] for y in (5, 9, 7, 12, 6, 8, 20, 10, 11) for x in range(10, 20)], np.int32)
    else:  # a column's second cell lies more than 128 cells up: it ends the chunk, the rest of the column does not
        cells = np.array([[x, y, 20] for x in range(10, 20) for y in (5, 140, 6, 100, 7)], np.int32)
    cells = np.ascontiguousarray(cells)
    assert sim.apply_brush(cells, STONE) == o.apply_brush(cells, STONE)
    same(sim, o, 2)
    sim.close()


# cells without water touch nothing but themselves and may come in any order: columns that reach as far below and
# above their first cell as one walk goes, and one row further, in air and with water at the bottom
@pytest.mark.parametrize("first", [60, 100, 20])
@pytest.mark.parametrize("order", ["listed", "down", "shuffled"])
def test_dry_columns_in_any_order(vf, orc, first, order):
    sim, o = pool(vf, orc, 200, 40)
    ys = [first] + [y for y in (first - 31, first - 32, first - 33, first + 95, first + 96, first - 1, first + 1, first + 40, first - 20, 39, 41) if 4 <= y < 200]
    if order == "down":
        ys = sorted(set(ys))[::-1]
    elif order == "shuffled":
        ys = np.random.default_rng(first).permutation(sorted(set(ys))).tolist()
    cells = np.array([[x, y, 20] for x in range(10, 20) for y in ys], np.int32)
    assert sim.apply_brush(cells, STONE) == o.apply_brush(cells, STONE)
    same(sim, o)
    cells = np.random.default_rng(7).permutation(sphere((24, 70, 24), 7))  # all dry
    cells = np.ascontiguousarray(cells)
    assert sim.apply_brush(cells, STONE) == o.apply_brush(cells, STONE)
    same(sim, o, 2)
    sim.close()
