"""Chunks that come and go on a live ring world, against the oracle: what the engine keeps of the cells (the
dense words) follows the chunks, also where a paste is refused after its slot was emptied."""
import ctypes as C

import numpy as np
import pytest

from conftest import assert_same_digest, oracle_for

pytestmark = pytest.mark.gpu
STONE, WATER = 3, 5


def flat(vf, ny=64):
    c = vf.World(128, ny, 128)
    c.fill_box(0, 0, 0, 127, 7, 127, STONE)
    return c


def block_over_the_border(vf, ny=64, **kw):
    """Two chunks with a block of water across x = 0."""
    ring = vf.World.ring(4, ny)
    for cx in (-1, 0):
        ring.ring_paste(flat(vf, ny), cx, 0)
    ring.fill_box(-20, 8, 40, 19, 30, 59, WATER)
    ring.fill_box(-3, 8, 45, 2, 12, 54, 0)
    return ring, vf.FluidSim(ring, **kw)


def refused_paste(vf, sim, grid, bricks, nbricks, bricks_y, cx, cz):
    grid, bricks = np.ascontiguousarray(grid, np.uint32), np.ascontiguousarray(bricks, np.uint8)
    return vf.lib().vf_fluid_ring_paste(sim.h, grid.ctypes.data_as(C.POINTER(C.c_uint32)), bricks.ctypes.data_as(C.POINTER(C.c_uint8)), nbricks,
                                        bricks_y, cx, cz)


@pytest.mark.parametrize("why", ["brick out of range", "atlas full"])
@pytest.mark.parametrize("evicted_before", [False, True])
def test_refused_paste_leaves_an_evicted_chunk(vf, orc, why, evicted_before):
    ring, sim = block_over_the_border(vf, atlas_bricks=400)
    o = oracle_for(orc, ring)
    for s in (sim, o):
        s.wake(-24, 7, 36, 23, 34, 63)
        s.tick(12)
    assert_same_digest(sim, o)
    if evicted_before:
        sim.ring_evict(0, 0)
    bumpy = flat(vf)
    for x in range(0, 128, 2):
        bumpy.fill_box(x, 8, 0, x, 40, 127, STONE)  # every brick of these layers is detailed
    grid, bricks, _ = bumpy.arrays()
    n = bricks.size // 512
    assert n > 1000
    rc = refused_paste(vf, sim, grid, bricks, 1 if why == "brick out of range" else n, bumpy.info.bricks_y, 0, 0)
    assert rc == (-1 if why == "brick out of range" else -2)
    o.ring_evict(0, 0)
    assert_same_digest(sim, o)
    for t in range(12):
        sim.tick()
        o.tick()
        assert_same_digest(sim, o, t)
        assert sim.partial_count() == o.partial_count()
    sim.close()


def test_chunks_come_and_go(vf, orc):
    """Six chunks under one block of water; chunks at the domain's corners, edges and middle leave and return
    while it flows, before and after the origin moves."""
    ring = vf.World.ring(4, 48)
    chunk = flat(vf, 48)
    where = [(cx, cz) for cx in (-1, 0, 1) for cz in (0, 1)]
    for cx, cz in where:
        ring.ring_paste(chunk, cx, cz)
    ring.fill_box(-12, 8, 116, 139, 20, 139, WATER)
    sim = vf.FluidSim(ring)
    o = oracle_for(orc, ring)
    for s in (sim, o):
        s.wake(-16, 7, 112, 143, 22, 143)
    grid, bricks, _ = chunk.arrays()
    shift = 0
    for t, (cx, cz) in enumerate(where + where[::-1]):
        if t == len(where):
            sim.shift(512, 0)
            o.ring_rebase(4, 0)
            o.shift(512, 0)
            shift = 4
        cx -= shift
        for s in (sim, o):
            s.ring_evict(cx, cz)
        assert_same_digest(sim, o)
        for s in (sim, o):
            s.tick(2)
        assert_same_digest(sim, o, t)
        xyz, vol = sim.partials()  # kept entries among them
        assert o.partial_count() == len(np.unique(xyz, axis=0)) and np.all(vol > 0)
        sim.ring_paste(chunk, cx, cz)
        o.ring_paste(grid, bricks, chunk.info.bricks_y, cx, cz)
        for s in (sim, o):
            s.tick(2)
        assert_same_digest(sim, o, t)
        xyz, vol = sim.partials()
        assert sim.partial_count() == o.partial_count() == len(np.unique(xyz, axis=0)) and np.all(vol > 0)
    sim.close()


def test_a_slot_changes_its_chunk(vf, orc):
    """Two slots a row, four chunks in the domain: a paste takes another chunk's slot, whose cells are outside then."""
    ring = vf.World.ring(2, 48)
    chunk = flat(vf, 48)
    for cx in (0, 3):
        ring.ring_paste(chunk, cx, 0)
    ring.fill_box(100, 8, 40, 127, 20, 60, WATER)
    ring.fill_box(384, 8, 40, 400, 20, 60, WATER)
    sim = vf.FluidSim(ring)
    o = oracle_for(orc, ring)
    for s in (sim, o):
        s.wake(96, 7, 36, 127, 22, 64)
        s.wake(384, 7, 36, 404, 22, 64)
    grid, bricks, _ = chunk.arrays()
    rain = np.array([[258 + i % 4, 30, 40 + i // 4] for i in range(32)], np.int32)
    for t, cx in enumerate((2, 1, 0, 3)):
        for s in (sim, o):
            s.tick(3)
        sim.ring_paste(chunk, cx, 0)
        o.ring_paste(grid, bricks, chunk.info.bricks_y, cx, 0)
        assert_same_digest(sim, o)
        for s in (sim, o):
            s.emit(rain, 0.6)
            s.tick(3)
        assert_same_digest(sim, o, t)
        assert sim.partial_count() == o.partial_count()
    sim.close()


def test_reset_between_chunks(vf, orc):
    """A reset takes the partial volumes, kept ones too, and leaves the materials."""
    ring, sim = block_over_the_border(vf)
    o = oracle_for(orc, ring)
    for s in (sim, o):
        s.wake(-24, 7, 36, 23, 34, 63)
        s.tick(14)
        s.ring_evict(0, 0)
        s.tick(2)
        s.set_partial(-5, 3, 45, 0.25)  # an entry in stone
        s.reset()
    assert_same_digest(sim, o)
    assert sim.partial_count() == o.partial_count() == len(sim.partials()[1]) == 0
    for s in (sim, o):
        s.wake(-24, 2, 36, 0, 34, 63)
    for t in range(6):
        sim.tick()
        o.tick()
        assert_same_digest(sim, o, t)
    chunk = flat(vf)
    grid, bricks, _ = chunk.arrays()
    sim.ring_paste(chunk, 0, 0)
    o.ring_paste(grid, bricks, chunk.info.bricks_y, 0, 0)
    for s in (sim, o):
        s.wake(-24, 2, 36, 23, 34, 63)
    for t in range(6):
        sim.tick()
        o.tick()
        assert_same_digest(sim, o, t)
    sim.close()
