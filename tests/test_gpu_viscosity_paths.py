"""Viscosity in the cells that its iterations do not write: a brick's cells outside the grid, in slots that have belonged to
other bricks. Against the oracle, bit for bit over whole active slots."""
import pytest

from slosh_b200 import _abi as A
from slosh_b200 import scenes

from parity import compare_state, pair

pytestmark = pytest.mark.gpu


def _scene(slosh, grid, iterations):
    s = scenes.base_settings(slosh.settings_default, grid, 40000)
    s.cell_size = 1.0 / max(grid)
    s.kinematic_viscosity, s.viscosity_iterations = 3e-4, iterations
    s.min_substeps = s.max_substeps = 2
    s.sparse_storage_budget = 0.6
    e = A.EmitRequest()
    e.shape, e.count = A.EMIT_SPHERE, 2500
    extent = [g * s.cell_size for g in grid]
    e.center[:] = [0.3 * extent[0], 0.6 * extent[1], 0.3 * extent[2]]
    e.extent[:] = [0.1, 0.0, 0.0]
    e.rotation[:] = [0.0, 0.0, 0.0, 1.0]
    e.velocity[:] = [6.0, 2.0, 7.0]  # through bricks that are freed behind it, into ones that the grid cuts
    e.speed_jitter = e.velocity_spread = 0.3
    return dict(settings=s, emits=[e], seed=3)


@pytest.mark.parametrize("iterations", [2, 4])
def test_cells_outside_the_grid_match_oracle(slosh, oracle_mod, iterations):
    sc = _scene(slosh, (37, 29, 43), iterations)
    g, o = pair(slosh, oracle_mod, sc)
    for f in range(16):
        fi = A.frame_input(sc["settings"], emits=sc["emits"] if f % 8 == 0 else [], delta_time=1.0 / 60.0)
        assert g.begin_frame(fi) == o.begin_frame(fi)
        for k in range(2):
            g.substep(k)
            o.substep(k)
            bad = compare_state(g, o).failures()
            assert not bad, (f, k, bad)
        g.end_frame()
        o.end_frame()
