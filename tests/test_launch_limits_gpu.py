"""A kernel's dynamic shared memory limit is the kernel's and the device's, not
the handle's or the thread's: a handle of a smaller shape that is created or
stepped in between, on the same or another thread, must not make the next
launch of a larger one fail."""

import threading

import numpy as np
import pytest

from pursuit_evasion_b200.batch import BatchSolve, BatchSolver
from pursuit_evasion_b200.reversible.free_dp import RelativeGrid
from pursuit_evasion_b200.reversible.relative_solver import RelativeSolver
from pursuit_evasion_b200.reversible.semilag import SemiLagrangianSolver
from pursuit_evasion_b200.reversible.world_dp import WorldGrid, WorldSolver
from tests.helpers import A3, bits

pytestmark = pytest.mark.gpu


def relative(precision, rows):
    # two tiles of one grid: the same kernel with more and less shared memory
    s = RelativeSolver(A3, RelativeGrid(33, 24, 11, 11, 8.0), local_precision=precision)
    s.set_tile(rows, 12)
    s.initialize()
    return s


def world(fast, grid):
    s = WorldSolver(A3, WorldGrid(*grid), fast=fast)
    s.init_square()
    return s


def semilag(grid):
    s = SemiLagrangianSolver(A3, RelativeGrid(*grid), mode="tube")
    s.set_kernel("tiled")
    s.initialize()
    return s


CASES = {
    "relative_float32": (lambda: relative("float32", 17), lambda: relative("float32", 4)),
    "relative_exact": (lambda: relative("float64", 17), lambda: relative("float64", 9)),
    "world_exact": (lambda: world(False, (9, 6, 3, 7, 3.5)),
                    lambda: world(False, (5, 4, 3, 7, 3.5))),
    "world_fast": (lambda: world(True, (9, 6, 3, 7, 3.5)),
                   lambda: world(True, (5, 4, 3, 7, 3.5))),
    "semilag_tiled": (lambda: semilag((33, 24, 7, 7, 6.0)),
                      lambda: semilag((13, 12, 7, 7, 3.0))),
}


def step(s):
    if isinstance(s, SemiLagrangianSolver):
        s.backup()
        s.residual()
    else:
        s.step(s.cfl_dt_limit if isinstance(s, RelativeSolver) else s.dt_limit)
        s.synchronize()


def result(s):
    return (s.value() if isinstance(s, SemiLagrangianSolver) else s.field()).copy()


@pytest.mark.parametrize("name", sorted(CASES))
def test_a_smaller_launch_on_another_thread_leaves_the_limit(name):
    big, small = CASES[name]
    with big() as alone:
        step(alone)
        step(alone)
        want = result(alone)
    failed = []
    with big() as a, small() as b:
        step(a)

        def other():
            try:
                step(b)
            except Exception as e:  # reported below
                failed.append(e)

        t = threading.Thread(target=other)
        t.start()
        t.join()
        step(a)
        got = result(a)
    assert not failed
    np.testing.assert_array_equal(bits(got), bits(want))


@pytest.mark.parametrize("precision", ["float64", "float32"])
def test_a_smaller_batch_created_later_leaves_the_limit(precision):
    wide = [BatchSolve(A3, RelativeGrid(49, 12, 5, 5, 4.0), 0.02)]
    narrow = [BatchSolve(A3, RelativeGrid(5, 8, 3, 3, 2.0), 0.02)]

    def solve(batch):
        batch.initialize()
        batch.run()
        batch.synchronize()
        return batch.field(0).copy()

    with BatchSolver(wide, local_precision=precision) as b:
        want = solve(b)
    with BatchSolver(wide, local_precision=precision) as a, \
            BatchSolver(narrow, local_precision=precision) as b:
        solve(b)
        np.testing.assert_array_equal(bits(solve(a)), bits(want))


def test_a_refused_batch_does_not_fail_the_next_call():
    """Rows of 2,300 positions exceed the float32 kernel's shared memory; the
    refusal leaves no error behind for the next handle's first check."""
    too_wide = [BatchSolve(A3, RelativeGrid(2300, 4, 3, 3, 8.0), 1e-4)]
    with pytest.raises(ValueError, match="do not fit"):
        BatchSolver(too_wide, local_precision="float32")
    with RelativeSolver(A3, RelativeGrid(9, 8, 3, 3, 2.0)) as s:
        s.initialize()
        step(s)
