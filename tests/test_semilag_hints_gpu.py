"""Stale order hints of the generic semi-Lagrangian backup: after many backups
each cell's hint is the optimum of that field, and the value that the backups
converge from moves it, so every backup here reads hints of another field.
They order the pairs only: each backup equals the oracle's and, bit for bit,
that of a fresh solver (neutral hints) on the same field."""

import numpy as np
import pytest

from pursuit_evasion_b200.reversible.free_dp import RelativeGrid
from pursuit_evasion_b200.reversible.semilag import SemiLagrangianSolver
from tests import oracle_lib
from tests.helpers import A3

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["tube", "min_time"])
@pytest.mark.parametrize("grid", [RelativeGrid(5, 4, 3, 3, 2.0), RelativeGrid(13, 7, 4, 5, 3.0)])
def test_backups_from_stale_hints_equal_the_oracle(oracle, grid, mode):
    omode = oracle_lib.SL_TUBE if mode == "tube" else oracle_lib.SL_MINTIME
    rng = np.random.default_rng(4)
    # noise: backups smooth it, and the optimum of most cells moves each time
    start = rng.uniform(0, 1, grid.states).astype(np.float32)
    with SemiLagrangianSolver(A3, grid, mode=mode) as s, \
            SemiLagrangianSolver(A3, grid, mode=mode) as fresh:
        s.set_kernel("generic")
        fresh.set_kernel("generic")
        cfg = oracle.sl_cfg(A3, grid, s.dt, omode)
        s.initialize(start)
        moved = []
        for _ in range(4):
            before = s.value().copy()
            fresh.initialize(before)  # resets its hints
            s.backup()
            fresh.backup()
            np.testing.assert_array_equal(s.value().view(np.uint32),
                                          fresh.value().view(np.uint32))
            want, up, ue = oracle.sl_backup(cfg, before.ravel().astype(np.float64), True)
            np.testing.assert_allclose(s.value().ravel(), want, atol=2e-5)
            moved.append((up, ue))
        changed = [np.mean((a[0] != b[0]) | (a[1] != b[1])) for a, b in zip(moved, moved[1:])]
        assert max(changed) > 0.05, changed  # the hints were wrong there
