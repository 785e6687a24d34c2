"""The sweep's counters come back under the names of what the kernel counts."""
import pytest

pytestmark = pytest.mark.gpu


def test_counters_name_what_is_counted(vf):
    wl = vf.Workload(1)  # the basin: many pressure searches
    sim = vf.FluidSim(wl.world(0), device=0)
    for b in wl.wakes(0):
        sim.wake(*map(int, b))
    sim.tick(8)
    p, s, st = sim.sweep_profile(), sim.sweep_stats(), sim.stats()
    assert set(p) == {"prepass", "rounds_and_pulls", "atlas_and_logs", "cta_searches", "wide_rounds", "cells", "searches", "rounds"}
    assert p["cells"] == st.cells_total > 0
    assert p["rounds"] == s["rounds"] > 8
    assert p["searches"] == s["searches"] > 0 and st.pull_success <= s["searches"]
    assert min(p["prepass"], p["atlas_and_logs"], p["wide_rounds"]) > 0
    assert p["rounds_and_pulls"] >= p["cta_searches"] + p["wide_rounds"]  # they are parts of it
    phases = sim.profile()
    assert set(phases) == {"drain", "sort", "sweep", "seed_commit", "level", "fifo_commit", "chg_commit", "mark_clear", "between"}
    assert sum(p[k] for k in ("prepass", "rounds_and_pulls", "atlas_and_logs")) <= phases["sweep"]
    sim.close()
