"""Every compiled form of the TMA-fed GEMM, entry for entry.

Tile width and stage count follow the number of CTAs against the number of SMs
(cvlbm_gemm_bf16), so the shapes here are counted in SMs: each reaches the form it
names, with fewer and more K slices than stages, stored and accumulated, into rows that
allow 16-byte accesses and rows that do not, with and without split K.  Operands and old
values are small integers: every product and every partial sum is an integer below 2^24,
exact in fp32 in any order, so C must equal the fp64 product.
"""

from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu

MAX_SPLITS = 64


def _form(M, N, K, split, sms):
    """(tile width, stages, splits) that the launch rule gives."""
    bn = 128 if N % 128 == 0 else 64
    tiles, splits = (M // 128) * (N // bn), 1
    while (split and splits < MAX_SPLITS and tiles * splits < 296 and (K // 64) % (2 * splits) == 0
           and K // 64 // (2 * splits) >= 4):
        splits *= 2
    if bn == 128 and tiles * splits < sms:
        bn = 64
    ctas = (M // 128) * (N // bn) * splits
    if bn == 128:
        return 128, 2 if 2 * sms < ctas <= 3 * sms else 3, splits
    return 64, 3 if ctas > sms else 6, splits


def _shapes(sms):
    odd = (sms + 3) | 1
    return {
        "128x3": (128, 128 * (sms + 9), 64, False),
        "128x3_slices": (256, 128 * (sms // 2 + 5), 448, False),
        "128x3_waves": (128, 128 * (3 * sms + 1), 128, False),
        "128x3_split": (128, 512, 16384, True),
        "128x2": (128, 128 * (2 * sms + 5), 320, False),
        "128x2_edge": (128, 128 * 3 * sms, 64, False),
        "128x2_split": (128, 768, 16384, True),
        "64x3": (128, 64 * odd, 64, False),
        "64x3_slices": (128, 64 * odd, 448, False),
        "64x3_narrowed": (128, 128 * (sms - 10), 256, False),
        "64x3_split": (128, 320, 16384, True),
        "64x6": (128, 192, 64, False),
        "64x6_slices": (256, 320, 832, False),
        "64x6_narrowed": (128, 640, 1024, False),
    }


@pytest.mark.parametrize("pad,offset", [(0, 0), (4, 0), (3, 0), (4, 1)])
@pytest.mark.parametrize("accumulate", [0, 1])
@pytest.mark.parametrize("name", sorted(_shapes(148)))
def test_every_form_is_exact_on_integers(name, accumulate, pad, offset, monkeypatch):
    import torch

    from test_gemm import _gemm

    monkeypatch.setenv("CVLBM_GEMM_LOADER", "tma")
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    M, N, K, split = _shapes(sms)[name]
    width, stages, splits = _form(M, N, K, split, sms)
    assert name.startswith(f"{width}x{stages}") and (splits > 1) == split

    g = torch.Generator(device="cuda").manual_seed(N + K)

    def ints(*shape):
        return torch.randint(-2, 3, shape, device="cuda", generator=g)

    A, B, C0 = ints(M, K), ints(N, K), ints(M, N).float()
    ldc = N + pad
    buf = torch.full((M * ldc + offset,), float("nan"), device="cuda")
    C = buf[offset:].view(M, ldc)[:, :N]
    if accumulate:
        C.copy_(C0)
    _gemm(A.to(torch.bfloat16), B.to(torch.bfloat16), C, accumulate=accumulate, split=split)
    want = A.double() @ B.double().T
    if accumulate:
        want = want + C0
    assert torch.equal(C.double(), want)
    if pad:
        assert bool(torch.isnan(buf[offset:].view(M, ldc)[:, N:]).all())
