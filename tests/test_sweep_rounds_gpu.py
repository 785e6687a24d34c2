"""The sweep's branches at their edges, against the oracle's one cell after another (state, FIFO, seeds and counters
after every tick): rounds run by one warp (up to 4 cells) and by all (lists past shared memory's 2048), searches
by one warp, by all warps and the ones told hopeless beforehand (open water, corners, floors, narrow CTAs),
the attempt budget, entries of solid cells, and what follows the order in which bricks get their slots."""
import hashlib

import numpy as np
import pytest

from conftest import assert_same_digest, oracle_for

pytestmark = pytest.mark.gpu
STONE, WATER = 3, 5


def run(sim, o, ticks):
    for t in range(ticks):
        sim.tick(1)
        o.tick(1)
        assert_same_digest(sim, o, t)


# isolated drops: one list of n cells in the first round, none of which wakes another
@pytest.mark.parametrize("n", [1, 4, 5, 64, 65, 2047, 2048, 2049, 4900])
def test_lists(vf, orc, n):
    w = vf.World(232, 24, 232)
    w.fill_box(0, 0, 0, 231, 3, 231, STONE)
    k = int(np.ceil(np.sqrt(n)))
    for i in range(n):
        x, z = 6 + 3 * (i % k), 6 + 3 * (i // k)
        w.fill_box(x, 12, z, x, 12, z, WATER)
    sim, o = vf.FluidSim(w, device=0), oracle_for(orc, w)
    for s in (sim, o):
        s.wake(0, 10, 0, 231, 14, 231)
    run(sim, o, 4)
    sim.close()


# water of a depth over a side, walled, drained through the floor in a corner or the middle
@pytest.mark.parametrize("warps", [0, 8])
@pytest.mark.parametrize("side,depth", [(6, 20), (14, 9), (14, 30), (30, 10), (30, 11), (30, 40), (45, 13)])
def test_deep_water(vf, orc, side, depth, warps):
    n, top = side + 4, depth + 20
    w = vf.World(n, top, n)
    w.fill_box(0, 0, 0, n - 1, 5, n - 1, STONE)
    for b in ((0, 0, n - 1, 1), (0, n - 2, n - 1, n - 1), (0, 0, 1, n - 1), (n - 2, 0, n - 1, n - 1)):
        w.fill_box(b[0], 4, b[1], b[2], top - 1, b[3], STONE)
    w.fill_box(2, 6, 2, n - 3, 5 + depth, n - 3, WATER)
    w.fill_box(2, 0, 2, 4, 5, 4, 0)
    w.fill_box(n // 2, 0, n // 2, n // 2 + 1, 5, n // 2 + 1, 0)
    w.fill_box(n - 5, 8, 2, n - 5, 7 + depth // 2, n - 3, STONE)  # a wall part of the way up
    sim, o = vf.FluidSim(w, device=0), oracle_for(orc, w)
    if warps:
        sim.set_sweep(2, 4 | 1 << 8 | warps << 16)
    for s in (sim, o):
        s.wake(0, 0, 0, n - 1, top - 1, n - 1)
    run(sim, o, 8)
    assert o.stats()["pull_attempts"] > 0
    sim.close()


# a free block of water: its sides run dry while its inside is deep
@pytest.mark.parametrize("size,height", [((12, 12), 12), ((9, 30), 24), ((26, 26), 26)])
def test_falling_block(vf, orc, size, height):
    w = vf.World(64, 64, 64)
    w.fill_box(0, 0, 0, 63, 3, 63, STONE)
    w.fill_box(10, 8, 10, 9 + size[0], 7 + height, 9 + size[1], WATER)
    sim, o = vf.FluidSim(w, device=0), oracle_for(orc, w)
    for s in (sim, o):
        s.wake(0, 0, 0, 63, 63, 63)
    run(sim, o, 10)
    sim.close()


def test_entries_of_solid_cells_and_partials_in_order(vf, orc):
    w = vf.World(70, 40, 70)  # several spans of the export, the last one cut short
    w.fill_box(0, 0, 0, 69, 3, 69, STONE)
    w.fill_box(5, 4, 5, 60, 9, 60, WATER)
    sim, o = vf.FluidSim(w, device=0), oracle_for(orc, w)
    rng = np.random.default_rng(1)
    for x, y, z in rng.integers((0, 0, 0), (70, 40, 70), (300, 3)).tolist():
        v = float(np.float32(rng.uniform(0.01, 0.99)))
        for s in (sim, o):
            s.set_partial(x, y, z, v)

    def check():
        xyz, vol = sim.partials()
        _, p = o.export_box(0, 0, 0, 70, 40, 70)
        z, y, x = np.nonzero(p > 0)
        assert np.array_equal(xyz, np.stack([x, y, z], 1)) and np.array_equal(vol.view(np.uint32), p[z, y, x].view(np.uint32))
        assert len(vol) == sim.partial_count()

    check()
    for s in (sim, o):
        s.wake(0, 0, 0, 69, 39, 69)
    run(sim, o, 3)  # a drained solid cell loses its entry
    check()
    sim.close()


def test_slots_do_not_change_from_run_to_run(vf):
    import torch

    from vfwater import proposal

    def features():
        h = hashlib.sha1()
        wl = vf.Workload(2, 0.125, 3)
        sim = vf.FluidSim(wl.world(0))
        for b in wl.wakes(0):
            sim.wake(*map(int, b))
        for _ in range(10):
            sim.tick(1)
            h.update(proposal.features(sim, torch)[0].cpu().numpy().tobytes())
        sim.close()
        return h.hexdigest()

    assert features() == features()


# cells side by side: one word of counts holds cells that finish and cells that are counted down
@pytest.mark.parametrize("width", [1, 2, 3, 4, 5, 7, 9])
def test_words_shared_by_finishing_and_waiting_cells(vf, orc, width):
    w = vf.World(96, 32, 96)
    w.fill_box(0, 0, 0, 95, 3, 95, STONE)
    for x in range(4, 90 - width, width + 3):
        w.fill_box(x, 10, 4, x + width - 1, 13, 80, WATER)
    sim, o = vf.FluidSim(w, device=0), oracle_for(orc, w)
    for s in (sim, o):
        s.wake(0, 8, 0, 95, 14, 95)
    run(sim, o, 4)
    sim.close()


# more cells below full than the budget has attempts: past it a cell does not wait for the cell two above it
def test_partial_block_past_the_attempt_budget(vf, orc):
    w = vf.World(90, 40, 90)
    w.fill_box(0, 0, 0, 89, 3, 89, STONE)
    sim, o = vf.FluidSim(w, device=0), oracle_for(orc, w)
    y, z, x = np.meshgrid(np.arange(12, 18), np.arange(8, 80), np.arange(8, 80), indexing="ij")
    cells = np.stack([x.ravel(), y.ravel(), z.ravel()], 1).astype(np.int32)
    for s in (sim, o):
        s.emit(cells, 0.9)
    run(sim, o, 4)
    assert sim.stats().pull_attempts >= 4096
    sim.close()


@pytest.mark.parametrize("n", [33, 128, 700])  # 96 x 97 .. 764 x 96 rows; tiles cut short, chunks of several tiles past 524,288 rows
def test_partials_in_order_over_chunks_of_rows(vf, n):
    ny = 65 if n < 700 else 760
    w = vf.World(n, ny, n)
    w.fill_box(0, 0, 0, n - 1, 3, n - 1, STONE)
    sim = vf.FluidSim(w, device=0, atlas_bricks=1 << 17)
    rng = np.random.default_rng(n)
    c = np.unique(np.concatenate([rng.integers((0, 4, 0), (n, ny, n), (9000, 3)), [[0, 4, 0], [n - 1, ny - 1, n - 1], [n - 1, 4, 0], [0, ny - 1, n - 1]],
                                  [[x, 9, n // 2] for x in range(n)], [[5, y, 7] for y in range(4, ny)]]), axis=0).astype(np.int32)
    assert len(sim.partials()[1]) == 0
    sim.emit(c, 0.3)
    xyz, vol = sim.partials()
    assert np.array_equal(xyz, c[np.lexsort((c[:, 0], c[:, 1], c[:, 2]))]) and np.all(vol == np.float32(0.3))
    assert sim.partial_count() == len(c)
    import ctypes as C

    take, total = len(c) // 3, C.c_uint64()  # fewer than there are: the first ones
    part, few = np.zeros((take, 3), np.int32), np.zeros(take, np.float32)
    assert vf.lib().vf_fluid_export_partials(sim.h, part.ctypes.data_as(C.POINTER(C.c_int32)), few.ctypes.data_as(C.POINTER(C.c_float)), take, C.byref(total)) == 0
    assert total.value == len(c) and np.array_equal(part, xyz[:take]) and np.all(few == np.float32(0.3))
    sim.close()
