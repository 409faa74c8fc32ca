"""Cells that the exact kernels recompute in the general form because their
fast evaluation met a value that is not finite, where the result is finite
after all: bit for bit the oracle's.

Relative stage: infinite values outside the local exit radius.  The exit resets
them, and a cell next to one has an infinite or undefined slope; the reference
then keeps its value (H < 0 is false) or moves it by its finite slopes.

8D stage: isolated values near the largest float.  Their difference quotients
overflow; the ENO selection drops an infinite one, the tube keeps the old value
or the floor takes over, and the cells beside are finite or not as the
reference's are.
"""

import ctypes

import numpy as np
import pytest

from pursuit_evasion_b200.reversible.free_dp import RelativeGrid
from pursuit_evasion_b200.reversible.relative_solver import RelativeSolver
from pursuit_evasion_b200.reversible.world_dp import WorldGrid, WorldSolver
from tests import oracle_lib
from tests.helpers import A3, bits

EXIT = 3.0


def relative_step(oracle, grid, order, field, arrival):
    """One step of the oracle with the local exit; the stages' own report of a
    cell that is not finite is left to the check of the result."""
    cfg = oracle.rel_cfg(A3, grid, order=order)
    dt = oracle.rel_cfl_limit(cfg)
    x = -grid.extent + np.arange(grid.positions) * (2 * grid.extent / (grid.positions - 1))
    out = np.broadcast_to(x[None, :] ** 2 + x[:, None] ** 2 > EXIT ** 2, grid.shape).reshape(-1)

    def stage(src, dst, blend):
        kept = arrival[out].copy()
        oracle.lib.po_rel_stage_f32(ctypes.addressof(cfg), src.ctypes.data, dst.ctypes.data,
                                    arrival.ctypes.data, dt, 0.0, blend, None)
        dst[out] = np.float32(EXIT)
        arrival[out] = kept

    other = np.full_like(field, np.nan)
    stage(field, other, 0)
    if order == 1:
        return other, dt
    stage(other, field, 1)
    return field, dt


def relative_case(grid, value):
    rng = np.random.default_rng(11)
    x = -grid.extent + np.arange(grid.positions) * (2 * grid.extent / (grid.positions - 1))
    far = np.broadcast_to(x[None, :] ** 2 + x[:, None] ** 2 > EXIT ** 2, grid.shape).reshape(-1)
    start = rng.normal(size=grid.states).astype(np.float32)
    start[far & (rng.random(grid.states) < 0.1)] = value
    return start


RELATIVE_GRIDS = [RelativeGrid(21, 8, 17, 16, 4.0), RelativeGrid(22, 13, 16, 14, 4.0)]


@pytest.mark.gpu
@pytest.mark.parametrize("grid", RELATIVE_GRIDS, ids=lambda g: f"{g.positions}x{g.headings}")
@pytest.mark.parametrize("order", [1, 2])
def test_relative_cells_beside_infinite_ones(oracle, grid, order):
    start = relative_case(grid, np.inf)
    arrival = np.where(start <= 0, np.float32(0), np.float32(np.nan)).astype(np.float32)
    with RelativeSolver(A3, grid, order=order, local_precision="float64") as s:
        s.set_exit(EXIT)
        s.initialize(start)
        s.step(s.cfl_dt_limit)
        field, got = s.field().reshape(-1), s.arrival().reshape(-1)
    want, _ = relative_step(oracle, grid, order, start, arrival)
    assert np.isfinite(want).all()
    np.testing.assert_array_equal(bits(field), bits(want))
    np.testing.assert_array_equal(np.isnan(got), np.isnan(arrival))
    held = ~np.isnan(arrival)
    np.testing.assert_array_equal(got[held], arrival[held])


@pytest.mark.gpu
@pytest.mark.parametrize("grid,size", [(WorldGrid(5, 4, 3, 3, 3.5), 1e38),
                                       (WorldGrid(6, 5, 4, 4, 3.5), 5e37),
                                       (WorldGrid(7, 4, 3, 5, 3.5), 2e37),
                                       (WorldGrid(5, 4, 3, 8, 3.5), 1e37)],
                         ids=lambda v: str(getattr(v, "e_speeds", "")))
@pytest.mark.parametrize("boundary,avoid", [("linear", True), ("legacy_signed", False)])
@pytest.mark.parametrize("sign", [1, -1])
def test_world_cells_whose_quotients_overflow(oracle, grid, size, boundary, avoid, sign):
    p, e = A3.pursuer, A3.evader
    cfg = oracle_lib.W8Cfg(grid.positions, grid.headings, grid.p_speeds, grid.e_speeds, 2,
                           int(boundary == "linear"), int(avoid), grid.extent,
                           A3.arena_half_width, A3.capture_radius, p.speed_min, p.speed_max,
                           e.speed_min, e.speed_max, p.acceleration, e.acceleration,
                           p.max_curvature, e.max_curvature, 0.8)
    rng = np.random.default_rng(7)
    a = rng.normal(size=grid.states).astype(np.float32)
    a[rng.choice(grid.states, grid.states // 500, replace=False)] = sign * size
    b = np.zeros_like(a)
    arrival = np.where(a <= 0, np.float32(0), np.float32(np.nan)).astype(np.float32)
    field, got = np.empty_like(a), np.empty_like(a)
    with WorldSolver(A3, grid, speed_boundary=boundary, avoid=avoid) as s:
        s.init_field(a)
        dt = s.dt_limit
        s.step(dt)
        for read, out in ((s.field, field), (s.arrival, got)):
            with pytest.raises(FloatingPointError):  # after the copy
                read(out)
    with np.errstate(all="ignore"):
        oracle.w8_stage(cfg, a, b, None, arrival, dt, 0.0)
        lost = ~np.isfinite(b)
        oracle.w8_stage(cfg, b, a, a, arrival, dt, 0.0)
    assert lost.any() and np.isfinite(a).mean() > 0.9
    known = ~np.isnan(a)
    np.testing.assert_array_equal(np.isnan(field), ~known)
    np.testing.assert_array_equal(bits(field)[known], bits(a)[known])
    np.testing.assert_array_equal(np.isnan(got), np.isnan(arrival))
    held = ~np.isnan(arrival)
    np.testing.assert_array_equal(got[held], arrival[held])
