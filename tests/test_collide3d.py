"""3-D fused collide kernel over step phases, sizes and laws, bit for bit.

The wavefront form (node_variant 3) keeps the moments in work items of their own and
the collision with its state in registers; node_variant 0 to 2 run k3_collide, which
forms the moments itself in a step with neither sweep nor repair.  Both evaluate the
same expressions, so runs agree exactly: kinematic intervals that mix all four kinds
of step, node counts that are no multiple of a block, laws with and without exp/log.
"""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,sweep,repair,model,source", [
    (19, 0, 0, "neo_hooke", "damping"),
    (22, 1, 1, "neo_hooke", "damping"),
    (21, 2, 3, "neo_hooke", "none"),
    (22, 3, 2, "gent", "damping"),
    (19, 0, 1, "svk", "damping"),
    (23, 1, 0, "mooney_rivlin", "damping"),
    (20, 2, 2, "log_neo_hooke", "constant"),
])
def test_collide_equals_the_wavefront_form(n, sweep, repair, model, source):
    from curved_lbm import workloads
    from curved_lbm.three_d import curved_boundary_warp3d as c3

    geom, mat, spec, kw = workloads.shell(n)
    if model != "neo_hooke":
        mat = c3.WarpHyperelasticMaterial3D.from_poisson(model, 0.25, mu=1.0)
    kw.update(local_displacement_interval=sweep, local_compatibility_interval=repair,
              source_mode=source)
    if source == "constant":
        kw["source_vector"] = tuple(1e-3 * k for k in range(1, 13))
    out = []
    for variant in (3, 0, 1, 2):
        s = c3.WarpSparseCurvedBoundaryLBM3D(geom, material=mat, boundary=spec, **kw)
        rng = np.random.default_rng(n)
        U = 1e-3 * rng.standard_normal((12, s.n_active))
        U[[3, 7, 11]] += 1.0
        s.initialize_from_numpy(U=U, displacement=1e-3 * rng.standard_normal((3, s.n_active)))
        s._select_variant(variant)
        s.run(1)
        s.run(6)
        out.append([s._host(t) for t in (s.f0, s.u_star, s.U, s.u, s.invalid)])
    assert np.isfinite(out[0][0]).all()
    for other in out[1:]:
        for a, b in zip(out[0], other):
            assert np.array_equal(a, b)
