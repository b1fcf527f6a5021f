"""2-D tile shapes at lattice sizes around their edges, bit for bit.

Heights 4, 8, 9, 10 and 16 rows of 32: lattices one node short of, on and past
multiples of them, odd rows, a lattice smaller than a tile.  Every shape evaluates the
same expressions, so a run must equal the split kernels' (variant 5), which have no
tiles.
"""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _solver(n, **kw):
    from curved_lbm import workloads
    from curved_lbm.two_d import curved_boundary_warp as c2

    geom, mat, spec, base = workloads.annulus(n)
    base.update(kw)
    s = c2.WarpCurvedBoundaryLBM2D(geom, material=mat, boundary=spec, **base)
    rng = np.random.default_rng(n)
    U = 1e-3 * rng.standard_normal((6, n, n))
    U[[2, 5]] += 1.0
    s.initialize_from_numpy(U=U, displacement=1e-3 * rng.standard_normal((2, n, n)))
    return s


@pytest.mark.parametrize("n", [31, 33, 63, 64, 71, 90, 97])
@pytest.mark.parametrize("kw", [{}, {"local_displacement_interval": 2,
                                     "local_compatibility_interval": 3},
                                {"local_displacement_interval": 0,
                                 "local_compatibility_interval": 0}])
def test_tile_shapes_equal_the_split_kernels(n, kw):
    ref = None
    for v in (5, 0, 1, 2, 3, 4, 6, 7, 8, 9, 10):
        s = _solver(n, **kw)
        s._select_variant(v)
        s.run(1)
        s.run(8)  # graph replay
        got = [s.numpy_field(k) for k in ("f0", "u_star", "U", "u", "invalid")]
        if ref is None:
            ref = got
            assert np.isfinite(ref[0]).all()
        for a, b in zip(ref, got):
            assert np.array_equal(a, b), v


def test_default_shape_follows_the_tile_count():
    import torch

    from curved_lbm.two_d import curved_boundary_warp as c2

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for n in (100, 600):
        s = _solver(n)
        few = (np.add.reduceat(np.add.reduceat(s.active_np, np.arange(0, n, 8), axis=0),
                               np.arange(0, n, 32), axis=1) > 0).sum() <= 2 * sms
        assert s.tile_variant == (c2.DEFAULT_TILE_VARIANT if few else c2.DEFAULT_TILE_VARIANT_LARGE)


def test_batch_runs_the_staged_tiles_and_refuses_the_others():
    from curved_lbm.batch import BATCH_DEFAULT_VARIANT, BatchedCurvedBoundaryLBM2D

    solo = [_solver(n) for n in (40, 57)]
    for s in solo:
        s.run(6)
    for v in (None, 8, 9, 10):
        group = [_solver(n) for n in (40, 57)]
        b = BatchedCurvedBoundaryLBM2D(group, tile_variant=v)
        assert b.tile_variant == (BATCH_DEFAULT_VARIANT if v is None else v)
        b.run(6)
        b.finish(refresh=False)
        for s, g in zip(solo, group):
            assert np.array_equal(s.numpy_field("f0"), g.numpy_field("f0"))
            assert np.array_equal(s.numpy_field("u_star"), g.numpy_field("u_star"))
    for v in (5, 6, 7, 11):
        with pytest.raises((RuntimeError, ValueError)):
            BatchedCurvedBoundaryLBM2D([_solver(40)], tile_variant=v)


@pytest.mark.parametrize("steps,kw", [(16, {}), (10, {}), (16, {"local_displacement_interval": 3}),
                                      (5, {})])
def test_autotune_replays_or_launches_and_restores_the_state(steps, kw):
    s = _solver(64, **kw)
    s.run(1)
    before = [s.numpy_field(k) for k in ("f0", "u_star")], s.time, s.steps
    times = s.autotune(steps=steps)
    assert len(times) == 11 and min(times.values()) > 0 and s.tile_variant in times
    assert s.use_graphs and not s._graphs
    assert (s.time, s.steps) == before[1:]
    for a, b in zip(before[0], (s.numpy_field("f0"), s.numpy_field("u_star"))):
        assert np.array_equal(a, b)
