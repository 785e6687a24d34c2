"""Levelling of small layers, several filled side by side, against the oracle's one after another: layers around the
64 cells and the 16 waiting entries that one warp fills, several seeds in one layer, films drained between levelled
layers, and a budget that runs out within a group. State, FIFO, seeds and level counters after every tick."""
import numpy as np
import pytest

from conftest import assert_same_digest, oracle_for

pytestmark = pytest.mark.gpu
STONE, WATER = 3, 5


def pits(vf, shapes, pitch, per_row, ny=16, depth=1):
    """A stone block with a pit of each shape (x, z extents) in its top, `depth` cells deep; their corners."""
    rows = (len(shapes) + per_row - 1) // per_row
    nx, nz = per_row * pitch + 2, rows * pitch + 2
    w = vf.World(nx, ny, nz)
    w.fill_box(0, 0, 0, nx - 1, 7, nz - 1, STONE)
    at = []
    for i, (sx, sz) in enumerate(shapes):
        x, z = 2 + pitch * (i % per_row), 2 + pitch * (i // per_row)
        w.fill_box(x, 8 - depth, z, x + sx - 1, 7, z + sz - 1, 0)
        at.append((x, z))
    return w, at


def both(vf, orc, w):
    return vf.FluidSim(w, device=0), oracle_for(orc, w)


def run(sim, o, ticks):
    for t in range(ticks):
        sim.tick(1)
        o.tick(1)
        assert_same_digest(sim, o, t)
        assert sim.stats().seed_count == len(o.queue()[1])


SHAPES = [(1, 2), (1, 63), (1, 64), (1, 65), (64, 1), (65, 1), (7, 9), (8, 8), (5, 13), (13, 5), (4, 16), (2, 32), (2, 33), (3, 21), (9, 7), (16, 4),
          (15, 15), (17, 17), (33, 2), (1, 1), (6, 10), (20, 20), (12, 5), (10, 6)]


@pytest.mark.parametrize("seed", [0, 1, 2])
def test_layers_around_the_limits(vf, orc, seed):
    """Uneven volumes in pits of every shape, all woken: every layer has many seeds, and a group holds large and small
    layers in the seeds' order."""
    rng = np.random.default_rng(seed)
    shapes = [SHAPES[i] for i in rng.permutation(np.resize(np.arange(len(SHAPES)), 40))]
    w, at = pits(vf, shapes, 67, 8)
    sim, o = both(vf, orc, w)
    for (x, z), (sx, sz) in zip(at, shapes):
        for dx in range(sx):
            for dz in range(sz):
                v = float(np.float32(rng.uniform(0.1, 0.95)))
                for s in (sim, o):
                    s.set_partial(x + dx, 7, z + dz, v)
    for s in (sim, o):
        for (x, z), (sx, sz) in zip(at, shapes):
            s.wake(x, 7, z, x + sx - 1, 7, z + sz - 1)
    run(sim, o, 12)
    assert o.stats()["level_cells"] > 1000
    sim.close()


def test_films_drain_between_levelled_layers(vf, orc):
    """Pits of water with a film of a few hundredths on it, which drains into the water below, in turn with pits that
    level to their average."""
    shapes = [(4, 4), (5, 5), (3, 7), (6, 2)] * 16
    w, at = pits(vf, shapes, 9, 8, depth=3)
    for i, (x, z) in enumerate(at):
        sx, sz = shapes[i]
        w.fill_box(x, 5, z, x + sx - 1, 6, z + sz - 1, WATER)
    sim, o = both(vf, orc, w)
    rng = np.random.default_rng(5)
    for i, ((x, z), (sx, sz)) in enumerate(zip(at, shapes)):
        lo, hi = ((0.01, 0.08), (0.2, 0.9))[i % 3 > 0]
        for dx in range(sx):
            for dz in range(sz):
                for s, v in zip((sim, o), [float(np.float32(rng.uniform(lo, hi)))] * 2):
                    s.set_partial(x + dx, 7, z + dz, v)
                if i % 3 == 0 and (dx + dz) % 2:
                    for s in (sim, o):
                        s.set_partial(x + dx, 6, z + dz, 0.9)
    for s in (sim, o):
        for _ in range(9):
            s.tick(1)
        for (x, z), (sx, sz) in zip(at, shapes):
            s.wake(x, 6, z, x + sx - 1, 7, z + sz - 1)
    run(sim, o, 14)
    assert o.stats()["drains"] > 20
    sim.close()


@pytest.mark.parametrize("side", [7, 8])  # 49 and 64 cells a pit, 1,024 and 784 pits: 50,176 cells
def test_budget_runs_out_within_a_group(vf, orc, side):
    """One seed in each pit of a levelling tick: 40,000 of the 50,176 cells are levelled in it, the rest in the next."""
    per_row = 32 if side == 7 else 28
    shapes = [(side, side)] * per_row**2
    w, at = pits(vf, shapes, side + 2, per_row)
    c = side // 2
    for x, z in at:
        w.fill_box(x, 7, z, x + side - 1, 7, z + side - 1, WATER)
    sim, o = both(vf, orc, w)
    for s in (sim, o):
        for x, z in at:
            for dx, dz in ((1, 0), (-1, 0), (0, 1), (0, -1)):
                s.set_partial(x + c + dx, 7, z + c + dz, 0.5)
        for _ in range(9):
            s.tick(1)
        for x, z in at:
            s.wake(x + c, 7, z + c, x + c, 7, z + c)
    run(sim, o, 1)
    assert 40000 <= sim.stats().last_level_cells < 40000 + 64 and sim.stats().level_round
    run(sim, o, 3)
    assert not sim.stats().level_round
    sim.close()
