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


def test_threads_with_calls_of_different_sizes(cuda_device):
    """The shared-memory limit of a kernel belongs to the process: small calls of one thread may not take it from the large
    ones of another (attention: 16 to 136 KB by the number of tokens; W4A4 layers: by tile width and ring depth)."""
    import threading

    from dimq_b200 import ops

    qkv = {t: torch.randn(2, t, 192, device="cuda").bfloat16() for t in (64, 512)}
    packed = ops.pack_bits(torch.randint(0, 16, (256, 768), device="cuda", dtype=torch.uint8), 4)
    book = torch.randn(16, device="cuda").half()
    rows = {m: torch.randn(m, 768, device="cuda") for m in (64, 2000)}

    def a4(m, n):
        return ops.dimq_linear_a4(rows[m], packed[:n * 384], book, 0.2, 7, None, n, 768)

    jobs = [lambda: ops.attention_qkv(qkv[64], 1), lambda: ops.attention_qkv(qkv[512], 1), lambda: a4(64, 64), lambda: a4(2000, 256)]
    want = [job() for job in jobs]
    torch.cuda.synchronize()
    errors = []

    def work(job, ref):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(300):
                    y = job()
                torch.cuda.current_stream().synchronize()
            if not torch.equal(y, ref):
                errors.append("wrong result")
        except Exception as e:          # noqa: BLE001 - reported below
            errors.append(repr(e))

    threads = [threading.Thread(target=work, args=a) for a in zip(jobs, want)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
