"""The pressure solvers' launch forms against the oracle, bit for bit after every substep, on grids whose bricks are cut
by the domain's faces and on ones with few and many active bricks."""
import pytest

from slosh_b200 import _abi as A
from slosh_b200 import scenes

from parity import pair, run_frames
from parity import compare_state

pytestmark = pytest.mark.gpu


def _scene(slosh, grid, solver, fill=(0.45, 0.6, 1.0), **settings):
    mn, dims = scenes.box_cells(grid, (0.0, 0.0, 0.0), fill)
    count = dims[0] * dims[1] * dims[2] * 8
    s = scenes.base_settings(slosh.settings_default, grid, count)
    s.cell_size = 1.0 / max(grid)
    s.pressure_solver = solver
    s.max_substeps = 2
    for k, v in settings.items():
        setattr(s, k, v)
    return dict(settings=s, emits=[scenes.fill_cells(mn, dims)], seed=5)


# one brick, an odd grid of cut bricks, a grid of 8-cell multiples, a longer one
@pytest.mark.parametrize("grid", [(8, 8, 8), (21, 17, 30), (32, 24, 40), (70, 41, 23)])
@pytest.mark.parametrize("iterations", [1, 20])
def test_rbgs_matches_oracle(slosh, oracle_mod, grid, iterations):
    sc = _scene(slosh, grid, A.SOLVER_RBGS, pressure_iterations=iterations, density_projection_iterations=iterations, sor_weight=1.7)
    g, o = pair(slosh, oracle_mod, sc)
    run_frames(g, o, sc, frames=3, tol=None)
    rg, ro = g.results(), o.results()
    # FP64 sums of the same FP32 terms in two orders
    assert rg.last_solve_true_rel_residual == pytest.approx(ro.last_solve_true_rel_residual, rel=1e-6)


# more bricks in the layout than the quarter-brick split takes: the first frame sweeps whole bricks
def test_rbgs_whole_bricks_match_oracle(slosh, oracle_mod):
    sc = _scene(slosh, (130, 96, 70), A.SOLVER_RBGS, pressure_iterations=3, density_projection_iterations=2, max_substeps=1)
    g, o = pair(slosh, oracle_mod, sc)
    run_frames(g, o, sc, frames=2, tol=None)


# The cluster form of the solve (few active bricks) and the launched form against the oracle: one and two tail levels,
# levels between level 0 and the tail, fixed counts and a tolerance, every preconditioner option, each storage precision.
@pytest.mark.parametrize("grid", [(16, 16, 16), (21, 17, 30), (64, 40, 33), (96, 72, 50)])
@pytest.mark.parametrize("settings", [
    dict(tolerance=0.0, pcg_iterations=3),
    dict(tolerance=1e-6, mg_smoothing_sweeps=2, mg_correction_scale=1.9, mg_coarse_iterations=4, mg_smoother_weight=1.15),
    dict(tolerance=1e-5, precision_mode=A.PRECISION_BF16_STORAGE, pcg_flexible=1, mg_smoothing_sweeps=3),
    dict(tolerance=1e-5, precision_mode=A.PRECISION_FP16_STORAGE, pcg_flexible=1, mg_smoother_weight=1.15),
    dict(tolerance=1e-12, max_iterations=2),
])
def test_mgpcg_forms_match_oracle(slosh, oracle_mod, grid, settings):
    sc = _scene(slosh, grid, A.SOLVER_MGPCG, **settings)
    g, o = pair(slosh, oracle_mod, sc)
    run_frames(g, o, sc, frames=2, tol=None)


# a layout of many bricks with few active ones: launched first, one cluster from the second frame on
def test_mgpcg_few_bricks_of_a_large_layout_match_oracle(slosh, oracle_mod):
    sc = _scene(slosh, (136, 136, 72), A.SOLVER_MGPCG, fill=(0.2, 0.25, 0.4), tolerance=1e-6, max_substeps=1)
    g, o = pair(slosh, oracle_mod, sc)
    run_frames(g, o, sc, frames=3, tol=None)


def _launches(g, fi):
    before = g.launch_count()
    g.step_frame(fi)
    return g.launch_count() - before


# Launches of a frame of one substep with 6 + 2 solver iterations: two cluster kernels and about 30 others, or more than ten an
# iteration. A level-4 tail (more than 4,096 cells at level 3) has no resident form and must not take the cluster.
@pytest.mark.parametrize("grid,cluster", [((128, 128, 120), True), ((136, 136, 136), False)])
def test_few_bricks_take_the_cluster_where_it_is_resident(slosh, oracle_mod, grid, cluster):
    sc = _scene(slosh, grid, A.SOLVER_MGPCG, fill=(0.1, 0.12, 0.1), pcg_iterations=6, max_substeps=1, mg_smoothing_sweeps=2)
    g, o = pair(slosh, oracle_mod, sc)
    run_frames(g, o, sc, frames=2, tol=None)
    n = _launches(g, A.frame_input(sc["settings"]))
    assert n < 50 if cluster else n > 90, n


def _drop_and_block(slosh):
    """A tank of 1,152 bricks with a drop in it that wakes 27 of them, and a block that wakes more than a cluster holds."""
    grid = (96, 96, 64)
    s = scenes.base_settings(slosh.settings_default, grid, 300000)
    s.pcg_iterations, s.min_substeps, s.max_substeps, s.mg_smoothing_sweeps = 6, 1, 1, 2
    s.gravity[:] = [0.0, 0.0, 0.0]
    return s, scenes.fill_cells((10, 10, 10), (4, 4, 4)), scenes.fill_cells((48, 16, 8), (40, 48, 16))


# A tank that is filled after a frame with few bricks is not solved by the few CTAs that those chose, however it is filled.
@pytest.mark.parametrize("how", ["frame", "emit", "upload", "write"])
def test_a_filled_tank_leaves_the_cluster(slosh, how):
    s, drop, block = _drop_and_block(slosh)
    full = slosh.Simulation(s)
    full.step_frame(A.frame_input(s, emits=[drop, block]))
    records = full.particles()
    g = slosh.Simulation(s)
    g.step_frame(A.frame_input(s, emits=[drop]))
    assert _launches(g, A.frame_input(s)) < 50
    if how == "emit":
        g.emit(block)
    elif how == "upload":
        g.upload_particles(records)
    elif how == "write":
        g.write("PARTICLES", records)
        g.write("BRICK_TOUCH", full.read("BRICK_TOUCH"))
    n = _launches(g, A.frame_input(s, emits=[block] if how == "frame" else []))
    assert int(g.read("ACTIVE_BRICKS")[0]) > 240 and n > 90, n


# An emitter that feeds the tank every frame, wherever it started, does not leave it.
@pytest.mark.parametrize("count", [40, 41])
def test_a_steady_emitter_keeps_the_cluster(slosh, count):
    s, drop, _ = _drop_and_block(slosh)
    e = A.EmitRequest()
    e.shape, e.count = A.EMIT_SPHERE, 40
    e.center[:] = [48 * s.cell_size, 48 * s.cell_size, 32 * s.cell_size]
    e.extent[:] = [14 * s.cell_size, 0.0, 0.0]  # 6^3 bricks with the layer around them
    e.rotation[:] = [0.0, 0.0, 0.0, 1.0]
    g = slosh.Simulation(s)
    g.step_frame(A.frame_input(s, emits=[drop, e]))
    for f in range(3):
        e.count = 40 if f == 0 else count
        assert _launches(g, A.frame_input(s, emits=[e])) < 50, f
    n = int(g.read("ACTIVE_BRICKS")[0])
    assert n + n // 16 <= 240  # what a cluster takes


# A tank that outgrows its cluster within a frame: a spray crosses brick boundaries, the cluster was chosen by the frame before,
# and the solve goes on over global memory. Tails at levels 1 to 3, several options each.
@pytest.mark.parametrize("grid,cells", [((32, 32, 32), 6), ((64, 64, 64), 14), ((104, 96, 100), 14)])
@pytest.mark.parametrize("settings", [
    dict(tolerance=0.0, pcg_iterations=3),
    dict(tolerance=1e-6, mg_smoothing_sweeps=2, mg_correction_scale=1.9, mg_coarse_iterations=4, mg_smoother_weight=1.15),
    dict(tolerance=1e-5, precision_mode=A.PRECISION_BF16_STORAGE, pcg_flexible=1, mg_smoothing_sweeps=3),
    dict(tolerance=1e-5, precision_mode=A.PRECISION_FP16_STORAGE, pcg_flexible=1, mg_smoother_weight=1.15),
])
def test_growth_within_a_frame_matches_oracle(slosh, oracle_mod, grid, cells, settings):
    s = scenes.base_settings(slosh.settings_default, grid, 8 * cells ** 3)
    s.cell_size = 1.0 / max(grid)
    s.max_frame_dt = 1.0 / 30.0
    for k, v in settings.items():
        setattr(s, k, v)
    e = scenes.fill_cells((9, 9, 9), (cells, cells, cells), velocity=tuple([5.0 * 60.0 * s.cell_size] * 3))  # 5 cells in a sixtieth
    e.velocity_spread, e.speed_jitter = 0.2, 0.4
    g, o = slosh.Simulation(s), oracle_mod.Oracle(s)
    bricks = []
    for f in range(3):
        s.min_substeps = s.max_substeps = 1 if f < 2 else 6
        fi = A.frame_input(s, emits=[e] if f == 0 else [], delta_time=1e-4 if f < 2 else 1.0 / 60.0)
        assert g.begin_frame(fi) == o.begin_frame(fi)
        for k in range(1 if f < 2 else 6):
            g.substep(k)
            o.substep(k)
            bad = compare_state(g, o).failures()
            assert not bad, (f, k, bad)
            bricks.append(int(g.read("ACTIVE_BRICKS")[0]))
        g.end_frame()
        o.end_frame()
        assert g.results().last_solve_iterations == o.results().last_solve_iterations
    ctas = next(c for c in range(4, 18, 2) if bricks[1] + bricks[1] // 16 <= 16 * (c - 1))
    assert ctas <= 16 and bricks[-1] > 16 * (ctas - 1), bricks


# levels 1 and 2 have too many tiles for the fused coarse passes, levels 3 and 4 do not
@pytest.mark.parametrize("settings", [
    dict(pcg_iterations=3),
    dict(pcg_iterations=3, mg_smoothing_sweeps=2, mg_correction_scale=1.9, mg_smoother_weight=1.15),
    dict(pcg_iterations=2, mg_smoothing_sweeps=2, precision_mode=A.PRECISION_BF16_STORAGE, pcg_flexible=1),
])
def test_fused_levels_below_launched_ones_match_oracle(slosh, oracle_mod, settings):
    grid = (97, 129, 2048)
    s = scenes.base_settings(slosh.settings_default, grid, 150000)
    s.cell_size = 1.0 / 64.0
    s.sparse_storage_budget = 0.05
    s.min_substeps = s.max_substeps = 1
    for k, v in settings.items():
        setattr(s, k, v)
    sc = dict(settings=s, emits=[scenes.fill_cells((30, 40, 1000), (24, 24, 30))], seed=1)
    g, o = pair(slosh, oracle_mod, sc)
    run_frames(g, o, sc, frames=2, tol=None)
