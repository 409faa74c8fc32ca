"""The exact 8D column kernel (csrc/world8d_column_exact.cu) against the
oracle's stage, bit for bit: every evader-speed count it is compiled for, both
speed boundaries and orders, one and several column groups, fields of noise,
of tied differences with signed zeros, with values too small for its quotients
(where a launch falls back to the range-checked ones), and values on both sides
of that bound."""

import numpy as np
import pytest

from pursuit_evasion_b200.reversible.world_dp import WorldGrid, WorldSolver
from tests import oracle_lib
from tests.helpers import A3

pytestmark = pytest.mark.gpu


def initial(kind, n):
    rng = np.random.default_rng(5)
    v = rng.normal(size=n)
    if kind == "plateau":
        v = np.round(2 * v) / 2
    elif kind == "tiny":
        v = v * 10.0 ** rng.integers(-44, 2, size=n)
    elif kind == "bound":
        v[rng.integers(0, n, n // 50)] = 2.0 ** -69.5
        v[rng.integers(0, n, n // 50)] = -(2.0 ** -70)
        v[rng.integers(0, n, n // 3)] = 0
    return v.astype(np.float32)


@pytest.mark.parametrize("grid", [WorldGrid(5, 4, 3, 3, 3.5), WorldGrid(6, 5, 4, 4, 3.5),
                                  WorldGrid(7, 4, 3, 5, 3.5), WorldGrid(5, 6, 5, 6, 3.5),
                                  WorldGrid(7, 5, 3, 7, 3.5), WorldGrid(10, 8, 3, 8, 3.5)],
                         ids=lambda g: f"{g.positions}x{g.headings}x{g.e_speeds}")
@pytest.mark.parametrize("order,boundary,avoid,kind", [
    (2, "linear", True, "noise"), (2, "legacy_signed", False, "plateau"),
    (2, "linear", False, "tiny"), (2, "legacy_signed", True, "bound"),
    (1, "linear", False, "plateau"), (1, "legacy_signed", False, "noise")])
def test_column_stage_equals_the_oracle(oracle, grid, order, boundary, avoid, kind):
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


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan, 3e38])
def test_column_stage_reports_values_that_are_not_finite(value):
    grid = WorldGrid(5, 4, 3, 3, 3.5)
    a = initial("noise", grid.states)
    a[grid.states // 3] = value
    a[grid.states // 3 + 1] = -value if np.isfinite(value) else a[0]
    with WorldSolver(A3, grid, avoid=False) as s:
        s.init_field(a)
        s.step(s.dt_limit)
        with pytest.raises(FloatingPointError):
            s.synchronize()
