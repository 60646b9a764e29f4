"""The density splat's three ways of adding a particle's moments (one shared tile, a tile in slabs, straight to global
memory) against the oracle on the same records: field, occupancy and mesh bit for bit (integer sums, so no tolerance)."""
import numpy as np
import pytest

import slosh_b200 as S

from test_gpu_surface import _compare

pytestmark = pytest.mark.gpu


def _records(grid, count, order, seed):
    """`count` records all over the domain, some dead, some at and beyond its faces."""
    rng = np.random.default_rng(seed)
    n = np.array(grid, np.float64)
    pos = rng.random((count, 3)) * n
    if order == "sorted":
        b = (pos // 4).astype(np.int64)
        pos = pos[np.argsort(b[:, 0] + 64 * (b[:, 1] + 64 * b[:, 2]), kind="stable")]
    edge = rng.integers(0, count, max(count // 50, 3))
    pos[edge, 0] = np.where(edge % 2, 0.0, n[0])
    rec = np.zeros(count, S.PARTICLE_DTYPE)
    rec["pos"] = (pos / max(grid)).astype(np.float32)
    rec["age"] = np.where(rng.random(count) < 0.1, -1.0, 1.0)
    rec["pos"][0] = -5.0 / max(grid)  # its kernel lies outside the field
    return rec


# counts around the CTA's 512 particles; kernels of one voxel up to the 4-voxel footprint (boxes of one tile, of several
# slabs, and of more slabs than are visited); records in sort order and in none
@pytest.mark.parametrize("count", [1, 511, 513, 4099])
@pytest.mark.parametrize("order", ["sorted", "random"])
@pytest.mark.parametrize("grid,res,smooth", [((24, 24, 24), 1.0, 2.0), ((40, 12, 21), 1.5, 0.5), ((20, 24, 28), 3.0, 6.0),
                                             ((120, 9, 33), 0.5, 3.0), ((96, 96, 40), 2.0, 1.0)])
def test_splat_paths_match_oracle(slosh, oracle_mod, grid, res, smooth, order, count):
    s = slosh.settings_default()
    s.grid_dim[:] = list(grid)
    s.cell_size = 1.0 / max(grid)
    s.particle_capacity = 8192
    rec = _records(grid, count, order, count)
    g, o = slosh.Simulation(s), oracle_mod.Oracle(s)
    for sim in (g, o):
        sim.upload_particles(rec)
    q = S.surface_params_default()
    q.field_resolution, q.surface_smoothing = res, smooth
    _compare(g, o, q)


# live records at infinite, NaN and far positions have no voxel: the field is the one without them, in kernels of three
# voxels, wider ones and ones that the footprint cuts
@pytest.mark.parametrize("res,smooth", [(1.0, 2.0), (1.5, 2.0), (1.5, 3.0), (3.0, 6.0)])
def test_splat_leaves_out_far_records(slosh, oracle_mod, res, smooth):
    grid = (24, 20, 28)
    s = slosh.settings_default()
    s.grid_dim[:] = list(grid)
    s.cell_size = 1.0 / max(grid)
    s.particle_capacity = 8192
    rec = _records(grid, 1500, "sorted", 5)
    far = [np.inf, -np.inf, np.nan, 1e30, -1e30] + [v * s.cell_size / res for v in (2.0 ** 31, -(2.0 ** 31), 2.0 ** 31 + 512.0, 1e9)]
    bad = np.zeros(3 * len(far) + 1, S.PARTICLE_DTYPE)
    bad["pos"] = 0.4
    for k, v in enumerate(far):
        for a in range(3):
            bad["pos"][3 * k + a, a] = v
    bad["pos"][-1] = np.inf
    bad["age"] = 1.0
    both = np.concatenate([rec[:700], bad, rec[700:]])
    q = S.surface_params_default()
    q.field_resolution, q.surface_smoothing = res, smooth
    g, o = slosh.Simulation(s), oracle_mod.Oracle(s)
    g.upload_particles(both)
    o.upload_particles(rec)
    _compare(g, o, q)


# more particles than a wave of CTAs with one particle per thread: two per thread, up to eight slabs
@pytest.mark.parametrize("order", ["sorted", "random"])
@pytest.mark.parametrize("res,smooth", [(1.0, 2.0), (1.5, 3.0)])
def test_splat_of_many_records_matches_oracle(slosh, oracle_mod, res, smooth, order):
    grid = (50, 64, 39)
    s = slosh.settings_default()
    s.grid_dim[:] = list(grid)
    s.cell_size = 1.0 / max(grid)
    s.particle_capacity = 200000
    rec = _records(grid, 190001, order, 7)
    g, o = slosh.Simulation(s), oracle_mod.Oracle(s)
    for sim in (g, o):
        sim.upload_particles(rec)
    q = S.surface_params_default()
    q.field_resolution, q.surface_smoothing = res, smooth
    _compare(g, o, q)
