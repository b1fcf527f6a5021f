"""3-D cut-link kernels on packed characteristic tables against the general ones.

The packed path (k3_link_gather_packed, k3_link_finish) and the path for tables of
any form (k3_link_gather, k3_link_prepare, k3_link_rows, k3_link_char) form the same
sums in the same order, so a run must agree bit for bit: per material law, Neumann
solver, value mode and mixed rows, at link counts that are no multiple of a block.
"""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _solver(n, model, spec_kw, **kw):
    from curved_lbm import workloads
    from curved_lbm.three_d import curved_boundary_warp3d as c3

    geom, mat, spec, base = workloads.shell(n)
    if model != "neo_hooke":
        extra = {"gent": {"gent_jm": 20.0}, "yeoh": {"yeoh_c2": 0.08, "yeoh_c3": 0.02}}.get(model, {})
        mat = c3.WarpHyperelasticMaterial3D.from_poisson(model, 0.25, mu=1.0, **extra)
    if spec_kw:
        spec = c3.CurvedBoundarySpec3D(**spec_kw)
    base.update(kw)
    s = c3.WarpSparseCurvedBoundaryLBM3D(geom, material=mat, boundary=spec, **base)
    rng = np.random.default_rng(n)
    U = 1e-3 * rng.standard_normal((12, s.n_active))
    U[[3, 7, 11]] += 1.0
    s.initialize_from_numpy(U=U, displacement=1e-3 * rng.standard_normal((3, s.n_active)))
    return s


TRACTION = dict(kind="neumann", value_mode=208, params=(0.05, 1.0),
                id_kinds={1: "neumann", 2: "dirichlet"}, id_value_modes={1: 208, 2: 0},
                id_params={1: (0.05, 1.0), 2: ()})
SINE2 = dict(kind="neumann", value_mode=203, params=(0.02, 0.5, 1.0),
             id_kinds={1: "neumann", 2: "neumann"}, id_value_modes={1: 203, 2: 0},
             id_params={1: (0.02, 0.5, 1.0), 2: ()})
MIXED = dict(TRACTION, id_component_kinds={1: ("neumann", "dirichlet", "neumann")})


@pytest.mark.parametrize("n,model,spec,kw", [
    (21, "neo_hooke", None, {}),
    (24, "neo_hooke", SINE2, {"neumann_solver": "energy"}),
    (24, "neo_hooke", MIXED, {"normal_jacobian": "finite_difference"}),
    (26, "gent", None, {}),
    (26, "svk", MIXED, {}),
    (25, "yeoh", SINE2, {}),
    (23, "sph_neo_hooke", None, {"source_mode": "none"}),
])
def test_packed_links_equal_general_links(n, model, spec, kw):
    states = []
    for packed in (True, False):
        try:
            s = _solver(n, model, spec, **kw)
        except (ValueError, TypeError) as exc:
            pytest.fail(str(exc))
        assert s._char_packed
        if not packed:
            s._problem.char_packed = 0
            s._problem.char_slot_lm = None
            s._problem.char_w_lm = None
        s.run(5)
        states.append([s._host(t) for t in (s.f0, s.U, s.u, s.u_star, s.char_state, s.link_Fb,
                                            s.link_Pb, s.link_bv, s.link_kind,
                                            s.link_component_kind)])
    assert np.isfinite(states[0][0]).all()
    for a, b in zip(*states):
        assert np.array_equal(a, b)


def test_tables_of_another_form_take_the_general_path():
    """User tables whose value weights share slots with gradient weights are not packed."""
    import torch

    from curved_lbm.three_d import curved_boundary_warp3d as c3

    w = torch.zeros((4, 64, 5), dtype=torch.float64)
    w[1:, :48], w[0, 48:] = 1.0, 2.0
    lm, packed = c3._link_major_weights(w)
    assert packed and lm.shape == (5, 48, 4)
    assert bool((lm[:, :, :3] == 1).all()) and bool((lm[:, :16, 3] == 2).all())
    assert not bool(lm[:, 16:, 3].any())
    w[0, 3, 2] = 0.5
    lm, packed = c3._link_major_weights(w)
    assert not packed and lm.shape == (5, 64, 4) and float(lm[2, 3, 0]) == 0.5
