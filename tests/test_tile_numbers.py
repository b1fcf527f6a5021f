"""Tile variants 6 and 7 with the tile lists that these numbers once stood for.

A caller of the C interface that kept 6 with tiles of 16 rows, or 7 with tiles of 8, runs
the fused step of that height: as many launches and the same bits as variants 0 and 2.
"""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("steps", [1, 4])
@pytest.mark.parametrize("old,now,rows", [(6, 0, 16), (7, 2, 8)])
def test_old_numbers_run_the_fused_step(old, now, rows, steps):
    from curved_lbm import _native
    from test_tiles2d import _solver

    got = []
    for number in (now, old):
        s = _solver(71)
        s.use_graphs = False
        s._select_variant(now)
        assert s._problem.tile_i == rows
        s._problem.tile_variant = number
        before = _native.launch_count()
        s.run(steps)
        got.append((_native.launch_count() - before, s.numpy_field("f0"), s.numpy_field("u_star")))
    assert got[0][0] == got[1][0]
    assert np.array_equal(got[0][1], got[1][1]) and np.array_equal(got[0][2], got[1][2])
