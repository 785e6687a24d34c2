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
