"""The tile shape of a batch that is given none: the first solver's if one was tuned or
selected for it, whatever its number, else the batch's default."""

from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu


def _solver():
    from curved_lbm import workloads
    from curved_lbm.two_d import curved_boundary_warp as c2

    geom, mat, spec, kw = workloads.annulus(40)
    return c2.WarpCurvedBoundaryLBM2D(geom, material=mat, boundary=spec, **kw)


@pytest.mark.parametrize("variant", [None, 0, 1, 3, 6, 9])
def test_batch_keeps_a_selected_shape(variant):
    from curved_lbm.batch import (BATCH_DEFAULT_VARIANT, BATCH_VARIANTS,
                                  BatchedCurvedBoundaryLBM2D)

    s = _solver()
    if variant is not None:
        s._select_variant(variant)
    b = BatchedCurvedBoundaryLBM2D([s])
    assert b.tile_variant == (variant if variant in BATCH_VARIANTS else BATCH_DEFAULT_VARIANT)


def test_batch_keeps_a_tuned_shape():
    from curved_lbm.batch import BatchedCurvedBoundaryLBM2D

    s = _solver()
    s.autotune(steps=8, variants=(1,))
    assert BatchedCurvedBoundaryLBM2D([s]).tile_variant == 1
