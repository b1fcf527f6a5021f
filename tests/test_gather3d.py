"""The three forms of the 3-D characteristic gather, bit for bit.

Packed tables (four lanes per link, k3_link_gather_packed), link-major tables of any
form (four lanes, k3_link_gather4) and the reference's table layout (16 lanes,
k3_link_gather) add a link's samples in slot order, so a run must agree; so must a run on
a given stencil whose gradient and value slots are mixed, which cannot be packed.
"""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(s, steps=5):
    s.run(steps)
    out = [s._host(t) for t in (s.f0, s.U, s.u, s.u_star, s.char_state, s.link_Fb, s.link_Pb)]
    assert np.isfinite(out[0]).all()
    return out


@pytest.mark.parametrize("n,model,spec", [(21, "neo_hooke", None), (26, "gent", None),
                                          (26, "svk", "mixed")])
def test_gather_forms_agree(n, model, spec):
    from test_links3d import MIXED, _solver

    spec = MIXED if spec else None
    want = _run(_solver(n, model, spec))  # packed

    s = _solver(n, model, spec)
    assert s._char_packed
    n_links = int(s.geometry.n_links)
    assert n_links % 32  # the last block of 32 links is ragged
    s._char_packed = False
    s._tables["char_w_lm"] = s._tables["char_w"].view(4, 64, n_links).permute(2, 1, 0).contiguous()
    s._problem = s._make_problem()
    assert s._problem.char_w_lm and s._problem.char_slot_lm and not s._problem.char_packed
    link_major = _run(s)

    s = _solver(n, model, spec)
    for name in ("char_slot_lm", "char_w_lm"):
        s._tables.pop(name)
    s._problem = s._make_problem()
    plain = _run(s)

    for a, b, c in zip(want, link_major, plain):
        assert np.array_equal(a, b) and np.array_equal(a, c)


@pytest.mark.parametrize("n,model", [(21, "neo_hooke"), (26, "yeoh")])
def test_given_stencil_with_mixed_slots(n, model):
    from test_links3d import _solver

    built = _solver(n, model, None)
    want = _run(built)
    order = np.r_[0:16, 48:64, 16:48]  # value samples between the gradient samples
    cs = built.characteristic_stencil
    cs = {"indices": np.asarray(cs["indices"])[order],
          "weights": np.asarray(cs["weights"])[:, order],
          "probe_modes": np.asarray(cs["probe_modes"])}
    s = _solver(n, model, None, characteristic_stencil=cs)
    assert not s._char_packed and s._problem.char_w_lm and not s._problem.char_packed
    for a, b in zip(want, _run(s)):
        assert np.array_equal(a, b)
