"""Host edits that run their list in parallel (voxel writes, emitters, carving) and the displacing
brush, against the oracle's sequential lists: voxels listed several times (within one chunk of 1024
and across chunks), lists around the chunk's length, bricks that are still uniform."""
import numpy as np
import pytest

from conftest import assert_same_state, oracle_for

pytestmark = pytest.mark.gpu
STONE, WATER = 3, 5


def lake(vf, orc, side=40, depth=9, top=28):
    w = vf.World(side, top, side)
    w.fill_box(0, 0, 0, side - 1, 3, side - 1, STONE)
    w.fill_box(0, 4, 0, side - 1, 3 + depth, side - 1, WATER)
    w.fill_box(10, 4, 10, 12, top - 1, 12, STONE)  # a pillar: columns that end at once
    w.compact()
    return vf.FluidSim(w, device=0), oracle_for(orc, w), (-1, 0, -1, side + 2, top + 1, side + 2)


def some_cells(rng, n, side=40, top=28, pool=0):
    """n cells in and just outside the world; `pool` > 0 draws them from that many, so that they repeat."""
    cells = np.stack([rng.integers(-1, side + 1, max(n, 1)), rng.integers(-1, top + 1, max(n, 1)), rng.integers(-1, side + 1, max(n, 1))], 1)
    cells = cells[rng.integers(0, pool, n)] if pool else cells[:n]
    return np.ascontiguousarray(cells, np.int32)


@pytest.mark.parametrize("n,pool", [(1, 0), (31, 3), (1023, 0), (1024, 200), (1025, 1), (2600, 700)])
def test_voxel_writes_in_list_order(vf, orc, n, pool):
    rng = np.random.default_rng(n)
    sim, o, box = lake(vf, orc)
    cells = some_cells(rng, n, pool=pool)
    mats = rng.choice([0, STONE, WATER, 7], n)
    before, _ = o.export_box(*box)
    sim.apply_voxel_edits([(int(x), int(y), int(z), int(m)) for (x, y, z), m in zip(cells, mats)])
    changed = set()
    for (x, y, z), m in zip(cells.tolist(), mats.tolist()):
        inside = 0 <= x < 40 and 0 <= y < 28 and 0 <= z < 40
        if inside and o.get_voxel(x, y, z) != m:
            changed.add((x, y, z))
        o.set_voxel(x, y, z, m)
    assert_same_state(sim, o, box)
    got = sim.download_changes()
    assert {tuple(c[:3]) for c in got.tolist()} == changed  # also voxels written back to what they held
    for x, y, z, m in got.tolist():
        assert m == o.get_voxel(x, y, z)
    sim.wake(0, 0, 0, 39, 27, 39)
    o.wake(0, 0, 0, 39, 27, 39)
    sim.tick(2)
    o.tick(2)
    assert_same_state(sim, o, box)
    sim.close()


@pytest.mark.parametrize("n,pool,amount", [(1, 0, 1.0), (40, 4, 0.3), (1024, 0, 0.25), (1025, 300, 0.4), (2100, 2, 0.0004)])
def test_emitters_in_list_order(vf, orc, n, pool, amount):
    rng = np.random.default_rng(n + 1)
    sim, o, box = lake(vf, orc)
    cells = some_cells(rng, n, pool=pool)
    for _ in range(2):  # the second time the cells are active and hold water
        sim.emit(cells, amount)
        o.emit(cells, amount)
        assert_same_state(sim, o, box)
        assert sim.partial_count() == o.partial_count()
    sim.tick(2)
    o.tick(2)
    assert_same_state(sim, o, box)
    sim.close()


@pytest.mark.parametrize("m", [0, STONE, WATER])
@pytest.mark.parametrize("n,pool", [(1, 0), (33, 5), (700, 0), (1500, 400)])
def test_brush_lists(vf, orc, n, pool, m):
    """Carving (in parallel) and placing (displacing water up its column, then to the sides)."""
    rng = np.random.default_rng(n + 2 + m)
    sim, o, box = lake(vf, orc)
    cells = some_cells(rng, n, top=16, pool=pool)
    for _ in range(2):
        assert sim.apply_brush(cells, m) == o.apply_brush(cells, m)
        assert_same_state(sim, o, box)
        assert sim.partial_count() == o.partial_count()
    sim.tick(2)
    o.tick(2)
    assert_same_state(sim, o, box)
    sim.close()


@pytest.mark.parametrize("depth", [1, 30, 31, 32, 33, 70])
def test_displaced_water_rises_past_a_full_column(vf, orc, depth):
    """The column above a displaced cell is read 32 cells at a time: surfaces on both sides of that."""
    w = vf.World(16, 104, 16)
    w.fill_box(0, 0, 0, 15, 3, 15, STONE)
    w.fill_box(0, 4, 0, 15, 3 + depth, 15, WATER)
    w.fill_box(4, 4 + depth, 4, 5, 4 + depth, 5, STONE)  # a lid: that column's water goes to the sides
    sim, o = vf.FluidSim(w, device=0), oracle_for(orc, w)
    for s in (sim, o):
        s.displace(8, 4, 8)
        s.displace(8, 4, 8)
        s.displace(4, 3 + depth, 4)
        s.displace(4, 3 + depth, 5)
        s.displace(15, 4, 0)
    assert_same_state(sim, o, (-1, 0, -1, 18, 105, 18))
    assert sim.partial_count() == o.partial_count()
    sim.close()


# one cell, or a few in turn, many times: over the levels where water shows and hides, until it is full or gone
@pytest.mark.parametrize("n", [2, 1023, 1024, 1025, 3000])
@pytest.mark.parametrize("cells", [1, 8])
@pytest.mark.parametrize("amount", [0.3, 0.013, 1e-4, 1e-7, -0.013, -0.3])
def test_emitters_of_the_same_cells(vf, orc, n, cells, amount):
    sim, o, box = lake(vf, orc)
    some = np.array([[20, 12, 20], [20, 13, 20], [5, 12, 5], [30, 20, 30], [11, 20, 11], [0, 4, 0], [20, 14, 20], [39, 27, 39]], np.int32)[:cells]
    lists = np.ascontiguousarray(np.resize(some, (n, 3)))
    for s in (sim, o):
        s.set_partial(20, 13, 20, 0.49)
        s.set_partial(5, 12, 5, 0.31)
    for _ in range(2):
        sim.emit(lists, amount)
        o.emit(lists, amount)
        assert_same_state(sim, o, box)
        assert sim.partial_count() == o.partial_count()
    assert all(m == o.get_voxel(x, y, z) for x, y, z, m in sim.download_changes().tolist())
    sim.tick(2)
    o.tick(2)
    assert_same_state(sim, o, box)
    sim.close()
