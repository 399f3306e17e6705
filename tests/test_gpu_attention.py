"""The packed-qkv attention kernel against a 64-bit softmax attention on the same 16-bit inputs."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("b,t,heads", [(1, 1, 1), (2, 63, 3), (1, 64, 12), (3, 65, 2), (1, 197, 12), (5, 256, 1), (1, 512, 2)])
def test_attention_qkv(cuda_device, b, t, heads, dtype):
    from dimq_b200 import ops

    gen = torch.Generator(device="cuda").manual_seed(t)
    qkv = (torch.randn(b, t, 3 * heads * 64, device="cuda", generator=gen) * 1.5).to(dtype)
    y = ops.attention_qkv(qkv, heads)
    q, k, v = qkv.double().view(b, t, 3, heads, 64).permute(2, 0, 3, 1, 4)
    want = (torch.softmax(q @ k.transpose(-1, -2) / 8, -1) @ v).transpose(1, 2).reshape(b, t, heads * 64)
    assert y.shape == want.shape and y.dtype == dtype
    # probabilities and the result are rounded to the element type: 2^-9 (2^-12) / sqrt(3) each
    rel = float((y.double() - want).norm() / want.norm())
    assert rel < (2.0 ** -8.5 if dtype == torch.bfloat16 else 2.0 ** -11.5), rel
    big = qkv.clone()
    big[:, :, :heads * 64] *= 60          # saturated softmax: scores of several hundred
    assert bool(ops.attention_qkv(big, heads).isfinite().all())


def test_attention_qkv_rejects(cuda_device):
    from dimq_b200 import ops

    for shape, heads in (((1, 513, 192), 1), ((1, 8, 96), 1), ((1, 8, 100), 1)):
        with pytest.raises(RuntimeError):
            ops.attention_qkv(torch.zeros(shape, device="cuda", dtype=torch.bfloat16), heads)
    with pytest.raises(RuntimeError):
        ops.attention_qkv(torch.zeros(1, 8, 192, device="cuda"), 1)
