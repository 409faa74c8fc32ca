"""The default tile of a solve: float32 keeps the widest even tile where no other
is estimated to be clearly faster, results do not depend on it, and (0, 0)
restores it."""

import numpy as np
import pytest

from pursuit_evasion_b200.reversible.free_dp import RelativeGrid
from pursuit_evasion_b200.reversible.relative_solver import RelativeSolver
from tests.helpers import A3, bits

pytestmark = pytest.mark.gpu


def even_tile(grid):
    """Up to 7 warps of 4-cell chunks with the fewest idle rows, at most 24
    headings in equal chunks."""
    chunks = (grid.positions + 3) // 4
    rows = min((r for r in range(1, grid.positions + 1) if r * chunks <= 224),
               key=lambda r: (-(-grid.positions // r) * r, -r))
    n = -(-grid.headings // 24)
    return rows, -(-grid.headings // n)


# grids whose even tile measured 6 to 22 % faster than the one that a coarser
# estimate takes
@pytest.mark.parametrize("shape,tile", [((40, 4, 20, 21), (20, 4)), ((40, 11, 24, 14), (20, 11)),
                                        ((26, 60, 23, 14), (26, 20)),
                                        ((65, 48, 21, 21), (13, 24))])
def test_grids_that_keep_the_even_tile(shape, tile):
    grid = RelativeGrid(*shape, 8.0)
    assert even_tile(grid) == tile
    with RelativeSolver(A3, grid, local_precision="float32") as s:
        assert s.tile == tile
        s.set_tile(4, tile[1])
        assert s.tile == (4, tile[1])
        s.set_tile(0, 0)
        assert s.tile == tile


@pytest.mark.parametrize("shape", [(17, 12, 7, 7), (41, 30, 13, 13), (31, 9, 5, 4)])
def test_grids_that_leave_it(shape):
    grid = RelativeGrid(*shape, 8.0)
    fields = []
    with RelativeSolver(A3, grid, local_precision="float32") as s:
        assert s.tile != even_tile(grid)
        for tile in (s.tile, even_tile(grid)):
            s.set_tile(*tile)
            s.initialize()
            for _ in range(3):
                s.step(s.cfl_dt_limit)
            fields.append(s.field().copy())
    np.testing.assert_array_equal(bits(fields[0]), bits(fields[1]))
