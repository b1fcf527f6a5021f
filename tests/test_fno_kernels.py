"""CUDA-core kernels of the warm-start surrogate at the sizes where they can go wrong.

Oracle: the same sums in plain PyTorch.  Where a kernel promises an order of
summation (over input channels, output channels or samples), the fp32 result
must equal the PyTorch loop in that order bit for bit (every product and sum
rounds separately: no FMA).  Sums over nodes are held to the fp32 bound
n eps sum|terms| of any order, against fp64.
"""

from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -24


def _lib():
    from curved_lbm import _native

    return _native, _native.load()


def _rand(seed, *shape):
    import torch

    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(*shape, device="cuda", generator=g)


# odd rows, one node, chunk of 128 with remainders 1 and 127, channel bounds 8/9/16/17/32
SIZES = [(1, 1, 1, 1), (2, 5, 7, 333), (4, 8, 32, 129), (3, 9, 12, 255), (4, 32, 12, 128),
         (2, 32, 16, 130), (1, 32, 17, 64), (4, 32, 32, 257)]


@pytest.mark.parametrize("B,ci,co,G", SIZES)
@pytest.mark.parametrize("act", [0, 1])
def test_layer_forward(B, ci, co, G, act):
    import torch

    nat, lib = _lib()
    x, W, b, s = _rand(1, B, ci, G), _rand(2, co, ci), _rand(3, co), _rand(4, B, co, G)
    for add in (True, False):
        z, y = torch.full((B, co, G), -9.0, device="cuda"), torch.empty(B, co, G, device="cuda")
        yb = torch.empty(B, co, G, device="cuda", dtype=torch.bfloat16)
        nat.check(lib.cvlbm_fno_layer_fwd(B, G, ci, co, nat.ptr(x), nat.ptr(W), nat.ptr(b),
                                          nat.ptr(s) if add else None, act, nat.ptr(z), nat.ptr(y),
                                          nat.ptr(yb), nat.stream_ptr(x.device)), "layer_fwd")
        ref = b[None, :, None].expand(B, co, G).clone()
        for i in range(ci):
            ref = ref + W[:, i][None, :, None] * x[:, i][:, None, :]
        if add:
            ref = ref + s
        assert torch.equal(z, ref)
        if act:  # erff and the two products: a few ulp of the result's size
            assert torch.allclose(y.double(), torch.nn.functional.gelu(z.double()), rtol=1e-6,
                                  atol=1e-6)
        else:
            assert torch.equal(y, z)
        assert torch.equal(yb, y.to(torch.bfloat16))


@pytest.mark.parametrize("B,ci,co,G", SIZES)
@pytest.mark.parametrize("act", [0, 1])
def test_layer_backward(B, ci, co, G, act):
    import torch

    nat, lib = _lib()
    dy, x, W, z = _rand(5, B, co, G), _rand(6, B, ci, G), _rand(7, co, ci), _rand(8, B, co, G)
    dx = torch.empty(B, ci, G, device="cuda")
    dzb = torch.empty(B, co, G, device="cuda", dtype=torch.bfloat16)
    dW, db = torch.empty(co, ci, device="cuda"), torch.empty(co, device="cuda")
    scr = torch.empty(int(lib.cvlbm_fno_pointwise_scratch(B, G, ci, co)), device="cuda")
    st = nat.stream_ptr(x.device)
    nat.check(lib.cvlbm_fno_layer_bwd(B, G, ci, co, nat.ptr(dy), nat.ptr(z) if act else None,
                                      nat.ptr(x), nat.ptr(W), nat.ptr(dx), nat.ptr(dzb), nat.ptr(dW),
                                      nat.ptr(db), nat.ptr(scr), st), "layer_bwd")
    dz = dy
    if act:
        dz = torch.empty_like(dy)
        nat.check(lib.cvlbm_fno_gelu_bwd(dy.numel(), nat.ptr(z), nat.ptr(dy), nat.ptr(dz), st),
                  "gelu_bwd")
    ref = torch.zeros(B, ci, G, device="cuda")
    for o in range(co):
        ref = ref + W[o][None, :, None] * dz[:, o][:, None, :]
    assert torch.equal(dx, ref)
    assert torch.equal(dzb, dz.to(torch.bfloat16))
    n = B * G
    w64 = torch.einsum("bog,big->oi", dz.double(), x.double())
    wabs = torch.einsum("bog,big->oi", dz.double().abs(), x.double().abs())
    assert bool(((dW.double() - w64).abs() <= (n + 1) * EPS * wabs).all())
    assert bool(((db.double() - dz.double().sum((0, 2))).abs()
                 <= n * EPS * dz.double().abs().sum((0, 2))).all())
    # accumulating dx through the older entry point
    dx2 = ref.clone()
    nat.check(lib.cvlbm_fno_pointwise_bwd(B, G, ci, co, nat.ptr(dz), nat.ptr(x), nat.ptr(W),
                                          nat.ptr(dx2), 1, nat.ptr(dW), nat.ptr(db), nat.ptr(scr),
                                          st), "pointwise_bwd")
    assert torch.equal(dx2, ref + ref)


@pytest.mark.parametrize("B,C,M", [(1, 1, 1), (4, 32, 64), (5, 32, 13), (9, 7, 17), (3, 16, 8)])
def test_spectral_mixing(B, C, M):
    import torch

    nat, lib = _lib()
    a, R, dbh = _rand(9, B, C, M), _rand(10, M, C, C), _rand(11, B, C, M)
    bh = torch.empty(B, C, M, device="cuda", dtype=torch.bfloat16)
    da, dR = torch.empty_like(bh), torch.empty_like(R)
    st = nat.stream_ptr(a.device)
    nat.check(lib.cvlbm_fno_spec_mix_fwd(B, C, M, nat.ptr(a), nat.ptr(R), nat.ptr(bh), st), "mix")
    nat.check(lib.cvlbm_fno_spec_mix_bwd(B, C, M, nat.ptr(a), nat.ptr(dbh), nat.ptr(R), nat.ptr(da),
                                         nat.ptr(dR), st), "mix_bwd")
    f, g = torch.zeros(B, C, M, device="cuda"), torch.zeros(B, C, M, device="cuda")
    for i in range(C):
        f = f + a[:, i][:, None, :] * R[:, i].t()[None]
        g = g + R[:, :, i].t()[None] * dbh[:, i][:, None, :]
    assert torch.equal(bh, f.to(torch.bfloat16))
    assert torch.equal(da, g.to(torch.bfloat16))
    r = torch.zeros_like(R)
    for b in range(B):
        r = r + a[b].t()[:, :, None] * dbh[b].t()[:, None, :]
    assert torch.equal(dR, r)


@pytest.mark.parametrize("B,G", [(1, 64), (4, 65536 // 12 + 5)])
def test_masked_loss(B, G):
    import torch

    nat, lib = _lib()
    y, t, w = _rand(12, B, 12, G), _rand(13, B, 12, G), _rand(14, 12).abs()
    mask = (_rand(15, B, G) > 0.3).float()
    out = []
    for mean in (False, True):
        dy, part = torch.empty_like(y), torch.empty(256, device="cuda")
        args = [B, 12, G, nat.ptr(y), nat.ptr(t), nat.ptr(mask), nat.ptr(w)]
        msum = mask.sum()
        inv = 1.0 / max(float(msum) * 12, 1.0)
        fn = lib.cvlbm_fno_mse_mean if mean else lib.cvlbm_fno_mse
        nat.check(fn(*args, nat.ptr(msum) if mean else inv, nat.ptr(dy), nat.ptr(part), 256,
                     nat.stream_ptr(y.device)), "mse")
        out.append((dy, part))
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])
    e = y.double() - t.double()
    m = mask.double()[:, None] * w.double()[None, :, None]
    assert torch.allclose(out[0][0].double(), 2 * m * e * inv, rtol=6 * 2 ** -23, atol=1e-12)
    loss = float((m * e * e).sum() * inv)
    assert abs(float(out[0][1].double().sum()) - loss) <= (e.numel() / 65536 + 16) * 2 ** -23 * loss


def test_adam_over_a_list_equals_adam_per_tensor():
    import ctypes as C

    import torch

    nat, lib = _lib()
    sizes = [1, 12, 1023, 1024, 1025, 5000] + [33] * 30  # more tensors than one launch holds
    p, g, m, v = ([_rand(20 + k + 50 * j, n).abs() for k, n in enumerate(sizes)] for j in range(4))
    q, mq, vq = ([t.clone() for t in lst] for lst in (p, m, v))
    st = nat.stream_ptr(p[0].device)
    hyper = (1e-3, 0.9, 0.999, 1e-8)
    for k, n in enumerate(sizes):
        nat.check(lib.cvlbm_fno_adam(n, nat.ptr(p[k]), nat.ptr(g[k]), nat.ptr(m[k]), nat.ptr(v[k]),
                                     *hyper, st), "adam")
    tab = [(C.c_void_p * len(sizes))(*[t.data_ptr() for t in lst]) for lst in (q, g, mq, vq)]
    nat.check(lib.cvlbm_fno_adam_list(len(sizes), (C.c_int64 * len(sizes))(*sizes), *tab, *hyper, st),
              "adam_list")
    for a, b in zip(p + m + v, q + mq + vq):
        assert torch.equal(a, b)
