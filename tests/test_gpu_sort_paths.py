"""The spatial sort's forms (one tile in one CTA, few tiles whose histograms every CTA adds up, many tiles with a scanned
histogram) against numpy's stable argsort: records, permutation, key offsets and counts, live count, exactly."""
import numpy as np
import pytest

import slosh_b200 as S

pytestmark = pytest.mark.gpu


def _records(grid, count, seed, order):
    rng = np.random.default_rng(seed)
    rec = np.zeros(count, S.PARTICLE_DTYPE)
    pos = rng.random((count, 3)) * (np.array(grid, np.float64) + 2.0) - 1.0  # some beyond the faces
    if order == "one":
        pos[:] = np.array(grid) * 0.5
    rec["pos"] = (pos / max(grid)).astype(np.float32)
    rec["age"] = np.where(rng.random(count) < (0.0 if order == "live" else 0.2), -1.0, 1.0)
    if order == "dead":
        rec["age"] = np.nan
    rec["vel"] = rng.standard_normal((count, 3)).astype(np.float32)
    return rec


def _expected(rec, grid):
    h = np.float32(1.0 / max(grid))
    inv_h = np.float32(1.0) / h
    c = [np.clip(np.floor(rec["pos"][:, a] * inv_h).astype(np.int64), 0, grid[a] - 1) >> 2 for a in range(3)]
    s = [(g + 3) // 4 for g in grid]
    keys = s[0] * s[1] * s[2] + 1
    key = np.where(rec["age"] >= 0.0, c[0] + s[0] * (c[1] + s[1] * c[2]), keys - 1)
    perm = np.argsort(key, kind="stable").astype(np.uint32)
    counts = np.bincount(key, minlength=keys).astype(np.uint32)
    offsets = (np.cumsum(counts) - counts).astype(np.uint32)
    return h, keys, perm, counts, offsets


# counts around a warp, the one-CTA form's 4096, a tile of the others and the 64 tiles that are added up; 1, 8, 9 and 18 key bits
@pytest.mark.parametrize("count", [1, 31, 4096, 4097, 8193, 262_144])
@pytest.mark.parametrize("grid", [(4, 4, 4), (24, 24, 18), (37, 50, 21), (255, 256, 256)])
@pytest.mark.parametrize("order", ["random", "live", "one", "dead"])
def test_static_sort_forms(slosh, grid, count, order):
    torch = pytest.importorskip("torch")
    rec = _records(grid, count, count, order)
    h, keys, perm, _, offsets = _expected(rec, grid)
    src = torch.from_numpy(rec.view(np.int32).reshape(count, 12).copy()).cuda()
    out = torch.empty_like(src)
    # outputs one word off their allocation: the permutation holds the tiles' histograms, scanned by 16-byte words where it can
    p = torch.empty(count + 1, dtype=torch.int32, device="cuda")[1:]
    o = torch.empty(keys + 1, dtype=torch.int32, device="cuda")[1:]
    live = torch.empty(1, dtype=torch.int32, device="cuda")
    S.sort_particles_static(src.data_ptr(), out.data_ptr(), count, grid, h, p.data_ptr(), o.data_ptr(), live.data_ptr())
    torch.cuda.synchronize()
    assert np.array_equal(p.cpu().numpy().view(np.uint32), perm)
    assert np.array_equal(o.cpu().numpy().view(np.uint32), offsets)
    assert int(live[0]) == int(offsets[-1])
    assert np.array_equal(out.cpu().numpy(), rec.view(np.int32).reshape(count, 12)[perm])


# the context's sort, with counts, up to more tiles than are added up
@pytest.mark.parametrize("count", [5, 4097, 262_145, 700_001])
def test_context_sort_forms(slosh, count):
    grid = (64, 60, 44)
    rec = _records(grid, count, 7, "random")
    h, keys, perm, counts, offsets = _expected(rec, grid)
    s = slosh.settings_default()
    s.grid_dim[:] = list(grid)
    s.cell_size = h
    s.particle_capacity = count
    sim = S.Simulation(s)
    sim.upload_particles(rec)
    sim.sort_particles()
    assert np.array_equal(sim.read("SORT_PERM"), perm)
    assert np.array_equal(sim.read("SORT_OFFSETS"), offsets)
    assert np.array_equal(sim.read("SORT_COUNTS"), counts)
    assert int(sim.read("PARTICLE_COUNT")[0]) == int(offsets[-1])
    assert np.array_equal(sim.read("PARTICLES").view(np.uint32), rec[perm].view(np.uint32))
