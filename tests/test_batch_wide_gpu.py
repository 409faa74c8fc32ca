"""Batches with rows of more than 1,024 positions, which exceed one 4-cell
chunk per thread of a CTA: the float32 kernel splits the row over items, the
exact batch takes a cell per thread (csrc/relative5d_batch_exact.cu)."""

import numpy as np
import pytest

from pursuit_evasion_b200.batch import BatchSolve, BatchSolver
from pursuit_evasion_b200.reversible.free_dp import RelativeGrid
from pursuit_evasion_b200.reversible.relative_solver import RelativeSolver
from tests.helpers import A3, bits

pytestmark = pytest.mark.gpu

SMALL = BatchSolve(A3, RelativeGrid(18, 9, 5, 4, 3.0), 0.05)


def thin(positions, steps):
    """A batch of `steps` RK2 steps on 4 headings and 3 x 3 speeds, and a small
    solve beside it."""
    grid = RelativeGrid(positions, 4, 3, 3, 8.0)
    with BatchSolver([BatchSolve(A3, grid, 1.0)]) as b:
        horizon = (steps - 0.5) * b.info(0)["dt_limit"]
    return [BatchSolve(A3, grid, horizon), SMALL]


def run(solves, precision):
    with BatchSolver(solves, local_precision=precision) as b:
        b.initialize()
        b.run()
        b.synchronize()
        return [(b.field(i).copy(), b.arrival(i).copy(), b.stats(i))
                for i in range(len(solves))]


@pytest.mark.parametrize("positions", [1024, 1025, 1031])
def test_float32_rows_wider_than_a_cta_are_updated(positions):
    """Against the exact batch after one RK2 step.  The CFL rule bounds the sum
    over the axes of dt times speed over spacing by 0.8.  Stage 1 reads equal
    inputs below 16: its results differ by a rounding (2^-20 = 9.5e-7) and by
    ENO selections of equal size and unlike sign, whose terms are a few
    roundings of the input (0.8 * 3e-6): 3.4e-6.  Stage 2 takes differences of
    that, a slope erring by four times as much (0.8 * 4 * 3.4e-6), and its own
    selections, and averages with equal old values: below 1e-5; twice that
    is allowed."""
    solves = thin(positions, 1)
    fast, exact = run(solves, "float32")[0], run(solves, "float64")[0]
    assert np.isfinite(fast[0]).all()
    assert np.abs(fast[0].astype(np.float64) - exact[0]).max() <= 2e-5
    # one step moves the values in the last columns by far more than that
    x = np.linspace(-8.0, 8.0, positions)
    start = (np.hypot(x[None, :], x[:, None]) - A3.capture_radius).reshape(exact[0].shape[-2:])
    assert np.abs(exact[0] - start)[..., -4:].max() > 2e-4


def test_wide_and_small_float32_solves_share_a_launch():
    alone = run([SMALL], "float32")[0]
    together = run(thin(1025, 1), "float32")[1]
    np.testing.assert_array_equal(bits(alone[0]), bits(together[0]))
    np.testing.assert_array_equal(bits(alone[1]), bits(together[1]))


@pytest.mark.parametrize("rows", [None, 3])
def test_exact_batch_of_wide_rows_equals_the_single_grid(rows):
    solves = thin(1025, 2)
    with BatchSolver(solves) as b:
        if rows:
            b.set_tile(0, rows)
            b.set_tile(1, rows)
        b.initialize()
        b.run()
        b.synchronize()
        got = [(b.field(i).copy(), b.arrival(i).copy(), b.stats(i)) for i in range(2)]
    for solve, (field, arrival, stats) in zip(solves, got):
        with RelativeSolver(solve.config, solve.grid, local_precision="float64") as s:
            s.initialize()
            s.advance(solve.horizon)
            np.testing.assert_array_equal(bits(field), bits(s.field()))
            np.testing.assert_array_equal(bits(arrival), bits(s.arrival()))
            assert stats == s.stats()
