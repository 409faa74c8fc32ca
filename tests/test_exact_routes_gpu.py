"""Which kernels the exact stages run, and the ones that few shapes reach: the
grids of the bit-for-bit tests are on the tiled and the column kernel, small
and unusual shapes a cell per thread, equal to the oracle there."""

import numpy as np
import pytest

from pursuit_evasion_b200.reversible.free_dp import RelativeGrid
from pursuit_evasion_b200.reversible.relative_solver import RelativeSolver
from pursuit_evasion_b200.reversible.world_dp import WorldGrid, WorldSolver
from tests import oracle_lib
from tests.helpers import A3, CONFIG1_GRID, CONFIG2_GRID, bits
from tests.test_relative_tiled_exact_gpu import GRIDS
from tests.test_recomputed_cells_gpu import RELATIVE_GRIDS
from tests.test_world_column_exact_gpu import initial

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid", GRIDS + RELATIVE_GRIDS + [RelativeGrid(33, 24, 11, 11, 8.0),
                                                           CONFIG2_GRID],
                         ids=lambda g: f"{g.positions}x{g.headings}")
@pytest.mark.parametrize("order", [1, 2])
def test_grids_of_the_tiled_tests_run_tiled(grid, order):
    with RelativeSolver(A3, grid, order=order, local_precision="float64") as s:
        assert s.exact_tiled


def test_small_wide_and_float32_solves_do_not():
    with RelativeSolver(A3, CONFIG1_GRID, local_precision="float64") as s:
        assert not s.exact_tiled
    with RelativeSolver(A3, RelativeGrid(1025, 4, 3, 3, 8.0), local_precision="float64") as s:
        assert not s.exact_tiled
    with RelativeSolver(A3, GRIDS[0], local_precision="float32") as s:
        assert not s.exact_tiled


@pytest.mark.parametrize("e_speeds", [3, 5, 8, 9])
def test_world_stages_run_by_columns_up_to_eight_evader_speeds(e_speeds):
    with WorldSolver(A3, WorldGrid(5, 4, 3, e_speeds, 3.5)) as s:
        assert s.exact_column == (e_speeds <= 8)


@pytest.mark.parametrize("order,boundary,avoid,kind", [
    (2, "linear", True, "noise"), (2, "legacy_signed", False, "plateau"),
    (2, "linear", False, "tiny"), (1, "legacy_signed", True, "noise")])
def test_world_cell_per_thread_stage_equals_the_oracle(oracle, order, boundary, avoid, kind):
    grid = WorldGrid(6, 5, 3, 9, 3.5)
    p, e = A3.pursuer, A3.evader
    cfg = oracle_lib.W8Cfg(grid.positions, grid.headings, grid.p_speeds, grid.e_speeds, order,
                           int(boundary == "linear"), int(avoid), grid.extent,
                           A3.arena_half_width, A3.capture_radius, p.speed_min, p.speed_max,
                           e.speed_min, e.speed_max, p.acceleration, e.acceleration,
                           p.max_curvature, e.max_curvature, 0.8)
    a = initial(kind, grid.states)
    b = np.zeros_like(a)
    arrival = np.where(a <= 0, np.float32(0), np.float32(np.nan)).astype(np.float32)
    with WorldSolver(A3, grid, order=order, speed_boundary=boundary, avoid=avoid) as s:
        s.init_field(a)
        dt, tau = s.dt_limit, 0.0
        for _ in range(2):
            s.step(dt)
            oracle.w8_stage(cfg, a, b, None, arrival, dt, tau)
            if order == 1:
                a, b = b, a
            else:
                oracle.w8_stage(cfg, b, a, a, arrival, dt, tau)
            tau += dt
        field, got = s.field().reshape(-1), s.arrival().reshape(-1)
    np.testing.assert_array_equal(field.view(np.uint32), a.view(np.uint32))
    np.testing.assert_array_equal(np.isnan(got), np.isnan(arrival))
    held = ~np.isnan(arrival)
    np.testing.assert_array_equal(got[held], arrival[held])


@pytest.mark.parametrize("boundary", ["linear", "legacy_signed"])
def test_world_fields_with_tiny_values_change_kernels(oracle, boundary):
    """Values below 2^-70 that the field starts with, or that a check finds, move
    the stages to a cell per thread, and back once they are gone; the results
    are the oracle's throughout.  Between checks the column kernel itself takes
    the general arithmetic."""
    grid = WorldGrid(7, 4, 3, 5, 3.5)
    p, e = A3.pursuer, A3.evader
    cfg = oracle_lib.W8Cfg(grid.positions, grid.headings, grid.p_speeds, grid.e_speeds, 2,
                           int(boundary == "linear"), 1, grid.extent, A3.arena_half_width,
                           A3.capture_radius, p.speed_min, p.speed_max, e.speed_min,
                           e.speed_max, p.acceleration, e.acceleration, p.max_curvature,
                           e.max_curvature, 0.8)

    def tiny(v):
        return bool(((v != 0) & (np.abs(v) < 2.0 ** -70)).any())

    with WorldSolver(A3, grid, speed_boundary=boundary) as s:
        dt = np.float32(s.dt_limit).item()
        for kind, check in (("noise", True), ("tiny", True), ("bound", True), ("bound", False),
                            ("one", True)):
            a = initial("noise" if kind == "one" else kind, grid.states)
            if kind == "one":
                a[a.size // 2] = 1e-30
            b = np.zeros_like(a)
            arrival = np.where(a <= 0, np.float32(0), np.float32(np.nan)).astype(np.float32)
            s.init_field(a)
            assert s.exact_column == (not tiny(a))
            tau, seen = 0.0, []
            for _ in range(4):
                s.step(dt)
                oracle.w8_stage(cfg, a, b, None, arrival, dt, tau)
                oracle.w8_stage(cfg, b, a, a, arrival, dt, tau)
                tau += dt
                if check:
                    s.synchronize()
                    seen.append(tiny(a))
                    assert s.exact_column == (not seen[-1])
            np.testing.assert_array_equal(bits(s.field().reshape(-1)), bits(a))
            got = s.arrival().reshape(-1)
            np.testing.assert_array_equal(np.isnan(got), np.isnan(arrival))
            if kind in ("noise", "one"):
                assert s.exact_column
