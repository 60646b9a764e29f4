"""P2G and G2P on records in every kind of place: sorted and not, beside and beyond the domain's faces, fast enough that an
advection step leaves its CTA's tile, dead, counts around a CTA. Against the oracle, bit for bit."""
import numpy as np
import pytest

import slosh_b200 as S
from slosh_b200 import _abi as A

from parity import compare_state

pytestmark = pytest.mark.gpu


def _records(grid, count, order, speed, seed):
    rng = np.random.default_rng(seed)
    n = np.array(grid, np.float64)
    pos = rng.random((count, 3)) * (n - 2.5) * np.array([0.6, 0.5, 1.0]) + 1.25
    if order == "sorted":
        b = (pos // 4).astype(np.int64)
        pos = pos[np.argsort(b[:, 0] + 64 * (b[:, 1] + 64 * b[:, 2]), kind="stable")]
    elif order == "outside":
        far = rng.random(count) < 0.1
        pos[far] = rng.random((int(far.sum()), 3)) * (n + 4.0) - 2.0
    rec = np.zeros(count, S.PARTICLE_DTYPE)
    rec["pos"] = (pos / max(grid)).astype(np.float32)
    rec["vel"] = (rng.standard_normal((count, 3)) * speed).astype(np.float32)
    half = rng.standard_normal((count, 10)).astype(np.float16)
    half[:, 9] = 0.0
    rec["c"] = half.view(np.uint32)
    rec["age"] = np.where(rng.random(count) < 0.05, -1.0, 1.0)
    return rec


@pytest.mark.parametrize("transfer", [A.TRANSFER_APIC, A.TRANSFER_FLIP])
@pytest.mark.parametrize("order,speed", [("sorted", 0.5), ("random", 0.5), ("outside", 0.5), ("sorted", 12.0)])
@pytest.mark.parametrize("count", [383, 385, 9000])
def test_transfers_match_oracle(slosh, oracle_mod, count, order, speed, transfer):
    grid = (30, 24, 21)
    s = slosh.settings_default()
    s.grid_dim[:] = list(grid)
    s.cell_size = 1.0 / max(grid)
    s.particle_capacity = 16384
    s.gravity[:] = [0.0, -9.81, 0.0]
    s.transfer_mode = transfer
    s.min_substeps = s.max_substeps = 2
    s.max_speed = 40.0
    g, o = slosh.Simulation(s), oracle_mod.Oracle(s)
    rec = _records(grid, count, order, speed, count)
    for sim in (g, o):
        sim.upload_particles(rec)
    fi = A.frame_input(s, delta_time=1.0 / 60.0)
    for _ in range(2):
        assert g.begin_frame(fi) == o.begin_frame(fi)
        for k in range(2):
            g.substep(k)
            o.substep(k)
            bad = compare_state(g, o).failures()
            assert not bad, bad
        g.end_frame()
        o.end_frame()


# the same records once sorted (the shared-memory tile, which unsorted ones do not take), and a frame after which they are
# in placement order again (the pool)
@pytest.mark.parametrize("density", [0, 1])
@pytest.mark.parametrize("order,speed", [("sorted", 0.5), ("outside", 0.5), ("sorted", 12.0)])
@pytest.mark.parametrize("count", [383, 385, 9000])
def test_apic_after_a_sort_matches_oracle(slosh, oracle_mod, count, order, speed, density):
    grid = (30, 24, 21)
    s = slosh.settings_default()
    s.grid_dim[:] = list(grid)
    s.cell_size = 1.0 / max(grid)
    s.particle_capacity = 16384
    s.min_substeps = s.max_substeps = 2
    s.max_speed = 40.0
    s.two_sided_density_projection = density
    s.sort_interval = 2
    g, o = slosh.Simulation(s), oracle_mod.Oracle(s)
    rec = _records(grid, count, order, speed, count)
    for sim in (g, o):
        sim.upload_particles(rec)
    fi = A.frame_input(s, delta_time=1.0 / 60.0)
    for f in range(3):
        if f == 2:
            rec = g.particles()[::-1].copy()
            for sim in (g, o):
                sim.upload_particles(rec)
        assert g.begin_frame(fi) == o.begin_frame(fi)
        for k in range(2):
            g.substep(k)
            o.substep(k)
            bad = compare_state(g, o).failures()
            assert not bad, bad
        g.end_frame()
        o.end_frame()


# a sorted spray (fewer than two particles a fluid cell) takes the pool from its second frame on
@pytest.mark.parametrize("density", [0, 1])
def test_sorted_spray_matches_oracle(slosh, oracle_mod, density):
    grid = (30, 24, 21)
    s = slosh.settings_default()
    s.grid_dim[:] = list(grid)
    s.cell_size = 1.0 / max(grid)
    s.particle_capacity = 16384
    s.two_sided_density_projection = density
    s.min_substeps = s.max_substeps = 1
    s.sort_interval = 1
    g, o = slosh.Simulation(s), oracle_mod.Oracle(s)
    rec = _records(grid, 1200, "random", 3.0, 9)
    for sim in (g, o):
        sim.upload_particles(rec)
    fi = A.frame_input(s, delta_time=1.0 / 120.0)
    for _ in range(3):
        assert g.begin_frame(fi) == o.begin_frame(fi)
        g.substep(0)
        o.substep(0)
        bad = compare_state(g, o).failures()
        assert not bad, bad
        g.end_frame()
        o.end_frame()
        assert g.results().live_particles < 2 * g.results().fluid_cells
