"""Attention backward at the edges of its tiles (128 stationary rows, 64 streamed rows per step).

Bound.  P, dS and O reach the tensor cores or the delta sum as bf16, each off by at most 2^-9 of
itself, and the outputs are rounded once more: relative to the 2-norm of a gradient that is
at most about 3 x 2^-9 from the operands, 2^-9 from O through delta and 2^-9 from the result,
together 5 x 2^-9 < 1e-2."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _reference(q, k, v, d_o, causal, scale):
    q, k, v = (t.double().permute(0, 2, 1, 3).requires_grad_(True) for t in (q, k, v))
    s = q @ k.transpose(-1, -2) * scale
    if causal:
        n = s.shape[-1]
        s = s.masked_fill(torch.ones(n, n, dtype=torch.bool, device=s.device).triu(1), -math.inf)
    (torch.softmax(s, -1) @ v).backward(d_o.double().permute(0, 2, 1, 3))
    return [t.grad.permute(0, 2, 1, 3) for t in (q, k, v)]


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("B,S,H", [(1, 1, 1), (2, 33, 3), (1, 63, 2), (1, 64, 2), (3, 65, 1), (1, 127, 2), (1, 128, 1),
                                   (2, 129, 2), (1, 191, 1), (1, 193, 2), (2, 333, 3), (1, 1000, 2)])
def test_lengths_off_the_tile_grid(B, S, H, D, causal):
    from luatorch_b200 import _C
    g = torch.Generator(device="cuda").manual_seed(S * 7 + D)
    qkv = torch.randn(B, S, 3, H, D, generator=g, device="cuda").bfloat16()
    q, k, v = qkv[:, :, 0], qkv[:, :, 1], qkv[:, :, 2]
    d_o = torch.randn(B, S, H, D, generator=g, device="cuda").bfloat16()
    scale = 1.0 / math.sqrt(D)
    o, lse = _C.flash_forward(q, k, v, causal, scale)
    packed = torch.full((B, S, 3, H, D), 7.0, device="cuda", dtype=torch.bfloat16)
    got = _C.flash_backward(q, k, v, o, lse, d_o, causal, scale, packed)
    assert _C.attention_device_error() == 0
    want = _reference(q, k, v, d_o, causal, scale)
    for name, a, b in zip(("dq", "dk", "dv"), got, want):
        # one key: dq and dk are exactly zero up to the rounding of O in delta
        floor = 2.0 ** -8 * math.sqrt(b.numel()) * scale * D if S == 1 else 0.0
        err = (a.double() - b).norm().item()
        assert err <= 1e-2 * b.norm().item() + floor, (name, err, b.norm().item())
    again = _C.flash_backward(q, k, v, o, lse, d_o, causal, scale, None)
    assert all(torch.equal(a, b) for a, b in zip(got, again))
