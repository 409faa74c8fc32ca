"""The tiled exact relative 5D stage (csrc/relative5d_tiled_exact.cu) against
the oracle's stage, bit for bit: every remainder of the x row by the 4-cell
chunk, rows that do not fill the last tile, both orders, the local exit, and
fields made of noise, of tied differences (plateaus, where the ENO selection
depends on the comparison's direction) and with values that are not finite.
The grids are large enough for the tiled kernel to be the chosen one."""

import numpy as np
import pytest

from pursuit_evasion_b200.reversible.free_dp import RelativeGrid
from pursuit_evasion_b200.reversible.relative_solver import RelativeSolver
from tests.helpers import A3

pytestmark = pytest.mark.gpu

GRIDS = [RelativeGrid(19, 12, 15, 13, 4.0), RelativeGrid(21, 8, 17, 16, 4.0),
         RelativeGrid(22, 13, 16, 14, 6.0), RelativeGrid(36, 9, 9, 9, 6.0),
         RelativeGrid(65, 13, 5, 6, 8.0)]


def initial(kind, n):
    rng = np.random.default_rng(3)
    if kind == "noise":
        return rng.normal(size=n).astype(np.float32)
    return (np.round(2 * rng.normal(size=n)) / 2).astype(np.float32)


@pytest.mark.parametrize("grid", GRIDS, ids=lambda g: f"{g.positions}x{g.headings}")
@pytest.mark.parametrize("order,kind,exit_radius", [(2, "noise", None), (2, "plateau", 3.0),
                                                    (1, "plateau", None)])
def test_tiled_exact_stage_equals_the_oracle(oracle, grid, order, kind, exit_radius):
    cfg = oracle.rel_cfg(A3, grid, order=order)
    start = initial(kind, grid.states)
    a, b = start.copy(), start.copy()
    arrival = np.where(a <= 0, np.float32(0), np.float32(np.nan)).astype(np.float32)
    x = -grid.extent + np.arange(grid.positions) * (2 * grid.extent / (grid.positions - 1))
    out = np.zeros(grid.states, bool)
    if exit_radius is not None:
        out = np.broadcast_to(x[None, :] ** 2 + x[:, None] ** 2 > exit_radius ** 2,
                              grid.shape).reshape(-1)

    def stage(src, dst, dt, t, blend):
        kept = arrival[out].copy()
        rc, _ = oracle.rel_stage_f32(cfg, src, dst, arrival, dt, t, blend)
        assert rc == 0
        if exit_radius is not None:
            dst[out] = np.float32(exit_radius)
            arrival[out] = kept

    with RelativeSolver(A3, grid, order=order, local_precision="float64") as s:
        s.set_exit(exit_radius)
        s.initialize(start)
        dt, t = s.cfl_dt_limit, 0.0
        for _ in range(2):
            s.step(dt)
            if order == 2:
                stage(a, b, dt, t, 0)
                stage(b, a, dt, t, 1)
            else:
                stage(a, b, dt, t, 0)
                a, b = b, a
            t += dt
        field, got_arrival = s.field().reshape(-1), s.arrival().reshape(-1)
    np.testing.assert_array_equal(field.view(np.uint32), a.view(np.uint32))
    np.testing.assert_array_equal(np.isnan(got_arrival), np.isnan(arrival))
    held = ~np.isnan(arrival)
    np.testing.assert_array_equal(got_arrival[held], arrival[held])


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
def test_values_that_are_not_finite_are_reported(value):
    grid = GRIDS[0]
    start = initial("noise", grid.states)
    start[grid.states // 3] = value
    with RelativeSolver(A3, grid, local_precision="float64") as s:
        s.initialize(start)
        s.step(s.cfl_dt_limit)
        with pytest.raises(FloatingPointError):
            s.synchronize()


@pytest.mark.parametrize("positions,headings,rows", [(17, 13, None), (18, 12, 18), (23, 7, 4),
                                                     (33, 25, None), (40, 9, 11), (5, 4, None)])
def test_tiled_batch_of_one_equals_the_single_grid(positions, headings, rows):
    """Few items, so short heading chunks; every row remainder; tiles that do
    not divide the rows or exceed what a CTA holds; two solves of unlike
    length share the launch."""
    from pursuit_evasion_b200.batch import BatchSolve, BatchSolver

    grid = RelativeGrid(positions, headings, 5, 4, 3.0)
    solves = [BatchSolve(A3, grid, 0.1), BatchSolve(A3, RelativeGrid(9, 8, 3, 3, 2.0), 0.03)]
    with BatchSolver(solves) as b:
        if rows:
            b.set_tile(0, rows)
        b.initialize()
        b.run()
        b.synchronize()
        got = [(b.field(i), b.arrival(i), b.stats(i)) for i in range(2)]
    for solve, (field, arrival, stats) in zip(solves, got):
        with RelativeSolver(solve.config, solve.grid, local_precision="float64") as s:
            s.initialize()
            s.advance(solve.horizon)
            np.testing.assert_array_equal(field.view(np.uint32), s.field().view(np.uint32))
            np.testing.assert_array_equal(arrival.view(np.uint32), s.arrival().view(np.uint32))
            assert stats == s.stats()


def test_exact_autotune_may_keep_the_default_tile(tmp_path):
    from dataclasses import replace

    from pursuit_evasion_b200.batch import BatchSolver, autotune, draw_batch

    solves = [replace(s, horizon=0.05) for s in draw_batch(4, count=2)]
    cache = tmp_path / "tiles.json"
    table = autotune.tune(solves, local_precision="float64", trial_steps=1, cache=cache)
    for bucket, rows in table.items():
        widths = [s.grid.positions for s in solves
                  if autotune.bucket_of(s.grid.positions) == bucket]
        assert rows in [0] + autotune.candidates(min(widths), "float64", max(widths))
    assert autotune.tune(solves, local_precision="float64", cache=cache) == table
    with BatchSolver(solves, local_precision="float64") as b:
        before = [b.tile(i) for i in range(len(solves))]
        autotune.apply(b, {bucket: 0 for bucket in table})
        assert [b.tile(i) for i in range(len(solves))] == before
