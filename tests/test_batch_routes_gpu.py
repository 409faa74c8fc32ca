"""Which kernel an exact batch runs, and that both give the single-grid solver's
bits: batches of small planes take a cell per thread, larger ones the tiled
kernel (every row remainder, heading chunks, tiles that do not divide the rows
or exceed what a CTA holds, two solves of unlike length)."""

import numpy as np
import pytest

from pursuit_evasion_b200.batch import BatchSolve, BatchSolver
from pursuit_evasion_b200.reversible.free_dp import RelativeGrid
from pursuit_evasion_b200.reversible.relative_solver import RelativeSolver
from tests.helpers import A3, bits

pytestmark = pytest.mark.gpu


def check(solves, tiled, rows=None):
    with BatchSolver(solves) as b:
        assert b.exact_tiled == tiled
        if rows:
            b.set_tile(0, rows)
            assert b.exact_tiled == tiled and b.tile(0) == rows
        b.initialize()
        b.run()
        b.synchronize()
        got = [(b.field(i), b.arrival(i), b.stats(i)) for i in range(len(solves))]
    for solve, (field, arrival, stats) in zip(solves, got):
        with RelativeSolver(solve.config, solve.grid, local_precision="float64") as s:
            s.initialize()
            s.advance(solve.horizon)
            np.testing.assert_array_equal(bits(field), bits(s.field()))
            np.testing.assert_array_equal(bits(arrival), bits(s.arrival()))
            assert stats == s.stats()


@pytest.mark.parametrize("positions,headings,p,e,rows", [
    (17, 13, 15, 13, None), (18, 12, 15, 13, 18), (23, 7, 15, 13, 4), (33, 25, 7, 7, None),
    (40, 9, 9, 9, 11), (49, 12, 7, 9, None)])
def test_tiled_batches(positions, headings, p, e, rows):
    check([BatchSolve(A3, RelativeGrid(positions, headings, p, e, 3.0), 0.08),
           BatchSolve(A3, RelativeGrid(9, 8, 3, 3, 2.0), 0.03)], True, rows)


@pytest.mark.parametrize("grids,rows", [([(12, 5, 14, 4)], None), ([(12, 5, 14, 4)], 5),
                                        ([(8, 46, 8, 3), (28, 5, 4, 6)], None),
                                        ([(9, 6, 6, 15)] * 3, 9), ([(5, 4, 3, 3)], None)])
def test_batches_of_small_planes(grids, rows):
    check([BatchSolve(A3, RelativeGrid(*g, 3.0), 0.04 + 0.02 * k)
           for k, g in enumerate(grids)], False, rows)


def test_default_tiles_follow_the_kernel():
    small = [BatchSolve(A3, RelativeGrid(24, 4, 3, 3, 3.0), 0.05)]
    large = [BatchSolve(A3, RelativeGrid(24, 24, 15, 15, 3.0), 0.05)]
    with BatchSolver(small) as b:
        assert not b.exact_tiled and b.tile(0) == 11  # 264 cells
    with BatchSolver(large) as b:
        assert b.exact_tiled and b.tile(0) == 24  # 144 chunks of 4 cells
    with BatchSolver(large, local_precision="float32") as b:
        assert not b.exact_tiled
