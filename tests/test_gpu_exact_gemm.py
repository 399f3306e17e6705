"""GPU parity of the fp32-grade tensor-core forms (W4A4 codes, fp32 activations) against 64-bit references.

Tolerance: both forms carry the operands to 2^-23 of each product and add fp32 partial sums of 256 k; the bound
used, 6e-7 of the result's norm, is four roundings of 2^-23 and a third over the 4.6e-7 that sequential fp32 FMAs
show at K = 768.
"""

from __future__ import annotations

import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu

REL = 6e-7


@pytest.fixture(scope="module")
def ops(cuda_device):
    from dimq_b200 import ops as _ops

    _ops.require_extension()
    return _ops


def _rel(y, want):
    return float((y.double() - want).norm() / want.norm())


def _weight(ops, n, k, bits, dtype, group_rows=None, seed=0):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    groups = 1 if group_rows is None else (n + group_rows - 1) // group_rows
    # codebooks of very different sizes, so that the scale of every group counts
    books = torch.randn(groups, 1 << bits, device="cuda", generator=gen) * 0.02
    books = (books * 4.0 ** torch.arange(groups, device="cuda").view(-1, 1)).to(dtype)
    idx = torch.randint(0, 1 << bits, (n, k), device="cuda", generator=gen, dtype=torch.uint8)
    rows = torch.arange(n, device="cuda") // (group_rows or n)
    return ops.pack_bits(idx, bits), books, torch.gather(books.double()[rows], 1, idx.long())


def _codes(x, scale, zp):
    q = torch.round(x.float() / torch.tensor(scale, device=x.device)) + zp
    return (q.clamp(0, 15) - zp).double() * torch.tensor(scale, dtype=torch.float32).double().item()


@pytest.mark.parametrize("m,k,n", [(1, 64, 4), (127, 192, 68), (129, 320, 132), (300, 1024, 1000), (1576, 768, 260)])
@pytest.mark.parametrize("book", [torch.float16, torch.bfloat16, torch.float32])
def test_linear_a4(ops, m, k, n, book):
    packed, books, w = _weight(ops, n, k, 4, book, seed=m)
    x = torch.randn(m, k, device="cuda").to(torch.float16 if m == 127 else torch.float32)
    bias = torch.randn(n, device="cuda")
    y = ops.dimq_linear_lut(x, packed, books.reshape(-1), 0.23, 7, bias, n, k)
    assert y.dtype == torch.float32 and ops.last_device_status() == 0
    assert _rel(y, _codes(x, 0.23, 7) @ w.t() + bias.double()) < REL


def test_linear_a4_long_sums(ops):
    # one-signed codes and codewords at K = 8192: sums far beyond 24 bits
    packed, books, w = _weight(ops, 128, 8192, 4, torch.float16, seed=3)
    books, w = books.abs(), w.abs()
    x = torch.rand(200, 8192, device="cuda") * 3
    y = ops.dimq_linear_lut(x, packed, books.reshape(-1), 0.2, 0, None, 128, 8192)
    assert _rel(y, _codes(x, 0.2, 0) @ w.t()) < REL


@pytest.mark.parametrize("epilogue,out", [("gelu", torch.float32), ("add_relu", torch.bfloat16), ("relu", torch.float16)])
def test_linear_a4_epilogues(ops, epilogue, out):
    m, k, n = 515, 256, 200
    packed, books, w = _weight(ops, n, k, 4, torch.float32, seed=9)
    x, res = torch.randn(m, k, device="cuda"), torch.randn(m, n, device="cuda").to(out)
    y = ops.dimq_linear_a4(x, packed, books.reshape(-1), 0.25, 8, None, n, k, out_dtype=out, epilogue=epilogue, residual=res)
    z = _codes(x, 0.25, 8) @ w.t()
    r = res.double()
    want = {"gelu": F.gelu(z) + r, "relu": z.relu() + r, "add_relu": (z + r).relu()}[epilogue]
    assert y.dtype == out and _rel(y, want) < {torch.float32: REL, torch.bfloat16: 2.0 ** -9, torch.float16: 2.0 ** -12}[out]


@pytest.mark.parametrize("batch,cin,cout,h,w_,ks,stride,pad", [
    (1, 64, 64, 1, 1, 1, 1, 0), (2, 64, 60, 7, 9, 3, 1, 1), (7, 128, 128, 28, 28, 3, 1, 1), (3, 64, 129, 15, 13, 3, 2, 1),
    (5, 192, 256, 14, 14, 1, 2, 0), (2, 512, 64, 7, 7, 3, 1, 1)])
@pytest.mark.parametrize("nhwc", [False, True])
@pytest.mark.parametrize("book", [torch.float16, torch.float32])
def test_conv2d_a4(ops, batch, cin, cout, h, w_, ks, stride, pad, nhwc, book):
    packed, books, w = _weight(ops, cout, cin * ks * ks, 4, book, seed=cin + ks)
    x = torch.randn(batch, cin, h, w_, device="cuda").relu_()
    if nhwc:
        x = x.contiguous(memory_format=torch.channels_last)
    bias = torch.randn(cout, device="cuda")
    y = ops.dimq_conv2d_lut(x, packed, books.reshape(-1), 0.28, 0, bias, (cout, cin, ks, ks), (stride, stride), (pad, pad),
                            (1, 1), 1)
    assert ops.last_device_status() == 0 and y.is_contiguous(memory_format=torch.channels_last if nhwc else torch.contiguous_format)
    want = F.conv2d(_codes(x.contiguous(), 0.28, 0), w.view(cout, cin, ks, ks), bias.double(), stride, pad)
    assert _rel(y, want) < REL


@pytest.mark.parametrize("m,k,n", [(9, 64, 4), (128, 128, 128), (197, 768, 1000), (130, 3072, 68)])
@pytest.mark.parametrize("bits,group_rows,book", [(4, None, torch.float32), (3, 16, torch.float32), (2, 128, torch.float16),
                                                  (4, 1, torch.bfloat16)])
def test_linear_f32(ops, m, k, n, bits, group_rows, book):
    if book == torch.float16 and n > 4 * 128:
        group_rows = 512                        # keeps the last group's codewords inside fp16
    if group_rows is not None and n // group_rows > 24:
        group_rows = (n + 23) // 24
    packed, books, w = _weight(ops, n, k, bits, book, group_rows, seed=m + bits)
    x = torch.randn(m, k, device="cuda") * 10.0 ** torch.linspace(-12, 12, m, device="cuda").view(-1, 1)
    bias = torch.randn(n, device="cuda")
    y = ops.dimq_linear_wq(x, packed, books, None, n, k, bits=bits, group_rows=group_rows)
    assert ops.last_device_status() == 0
    want = x.double() @ w.t()
    # row by row and group by group: neither a large row nor a large group may hide a small one
    err = (y.double() - want).view(m, n)
    gr = group_rows or n
    for g0 in range(0, n, gr):
        # the norm of |x| |w| / sqrt(k), not of the result: a row's few columns of one group may cancel, and rounding
        # errors follow the products.  The worst of 197 rows lies within 4 standard deviations.
        e = err[:, g0:g0 + gr].norm(dim=1)
        r = x.double().norm(dim=1) * w[g0:g0 + gr].norm() / k ** 0.5
        assert float((e / r).max()) < 4 * REL
    y2 = ops.dimq_linear_wq(x[:, :], packed, books, bias, n, k, bits=bits, group_rows=group_rows, epilogue="relu")
    # one row dominates this norm, and its few columns may cancel: rounding errors follow the products here too
    scale = float((x.double().norm() * w.norm() / k ** 0.5).clamp_min(1.0))
    assert float((y2.double() - (want + bias.double()).relu()).norm()) < REL * scale


def test_linear_f32_non_finite(ops):
    m, k, n = 40, 128, 64
    packed, books, w = _weight(ops, n, k, 4, torch.float32, seed=1)
    x = torch.randn(m, k, device="cuda")
    x[3, 5], x[7, 9], x[11, 2] = float("inf"), float("-inf"), float("nan")
    x[20] = 0.0
    x[21] *= 1e30
    y = ops.dimq_linear_wq(x, packed, books, None, n, k, bits=4)
    want = x @ w.float().t()
    assert torch.equal(y.isnan(), want.isnan()) and torch.equal(y.isinf(), want.isinf())
    ok = want.isfinite()
    assert torch.equal(y[~ok & ~want.isnan()].sign(), want[~ok & ~want.isnan()].sign())
    rows = ok.all(1)                                     # the rows without a non-finite element
    bound = 1e-5 * x[rows].double().norm(dim=1, keepdim=True) * w.norm(dim=1)
    assert bool(((y[rows] - want[rows]).abs() <= bound).all())
    # an infinite codeword
    bad = books.clone()
    bad[0, 3] = float("inf")
    hit = torch.isinf(bad.double()[torch.zeros(n, device="cuda", dtype=torch.long)].gather(
        1, torch.stack([(packed.view(n, -1) & 15), (packed.view(n, -1) >> 4)], 2).view(n, k).long())).any(1)
    x = torch.rand(m, k, device="cuda") + 0.5
    y = ops.dimq_linear_wq(x, packed, bad, None, n, k, bits=4)
    assert torch.equal(y.isinf().all(0), hit) and bool(y[:, ~hit].isfinite().all())


# ---- bf16 activations against an fp16 codebook: rows scaled into fp16 (GEMM), two terms in one MMA (convolution) --------
# Bound: the products are exact or carry 2^-17, the accumulators truncate: 3.7e-6 at K = 3072, 5.5e-6 at 4608.

@pytest.mark.parametrize("m,k,n", [(33, 768, 768), (197, 768, 1000), (400, 1024, 2048), (1024, 64, 8), (1025, 768, 328),
                                   (2000, 3072, 256), (9473, 256, 512)])
@pytest.mark.parametrize("bits,group_rows", [(4, None), (3, 128), (2, 1)])
def test_linear_bf16_rows_with_fp16_codebook(ops, m, k, n, bits, group_rows):
    if group_rows is not None and n // group_rows > 3:
        group_rows = n // 3                       # keeps the last group's codewords inside fp16
    packed, books, w = _weight(ops, n, k, bits, torch.float16, group_rows, seed=m + bits)
    x = (torch.randn(m, k, device="cuda") * 10.0 ** torch.linspace(-14, 14, m, device="cuda").view(-1, 1)).bfloat16()
    bias, res = torch.randn(n, device="cuda"), torch.randn(m, n, device="cuda")
    y = ops.dimq_linear_wq(x, packed, books, None, n, k, bits=bits, group_rows=group_rows)
    want = x.double() @ w.t()
    r = x.double().norm(dim=1) * w.norm() / k ** 0.5
    assert ops.last_device_status() == 0 and float(((y.double() - want).norm(dim=1) / r).max()) < 1.2e-5
    mm = min(m, 1024)
    y = ops.dimq_linear_wq(x[:mm], packed, books, bias, n, k, bits=bits, group_rows=group_rows, epilogue="relu",
                           residual=res[:mm])
    z = (want[:mm] + bias.double()).relu() + res[:mm].double()
    assert float((y.double() - z).norm() / z.norm()) < 1.2e-5


def test_linear_bf16_rows_non_finite(ops):
    m, k, n = 1100, 128, 64
    packed, books, w = _weight(ops, n, k, 4, torch.float16, seed=5)
    x = torch.randn(m, k, device="cuda").bfloat16()
    x[3, 5], x[700, 9], x[1099, 2] = float("inf"), float("-inf"), float("nan")
    x[20] = 0.0
    y = ops.dimq_linear_wq(x, packed, books, None, n, k, bits=4)
    want = x.float() @ w.float().t()
    assert torch.equal(y.isnan(), want.isnan()) and torch.equal(y.isinf(), want.isinf())
    assert bool((y[20] == 0).all())


@pytest.mark.parametrize("cout", [8, 64, 72, 128, 136, 256])
@pytest.mark.parametrize("cin,ks,stride,size", [(64, 3, 1, 28), (128, 1, 2, 28), (64, 1, 1, 33)])
def test_conv2d_two_terms(ops, cout, cin, ks, stride, size):
    packed, books, w = _weight(ops, cout, cin * ks * ks, 4, torch.float16, seed=cout + ks)
    x = torch.randn(9, cin, size, size, device="cuda").bfloat16().contiguous(memory_format=torch.channels_last)
    bias = torch.randn(cout, device="cuda")
    wshape = (cout, cin, ks, ks)
    y = ops.dimq_conv2d_wq(x, packed, books.reshape(-1), bias, wshape, stride, ks // 2, bits=4,
                           packed_khwc=ops.conv_prepack(packed, wshape, 4))
    want = F.conv2d(x.double().contiguous(), w.view(wshape), bias.double(), stride, ks // 2)
    assert ops.last_device_status() == 0 and _rel(y, want) < 1.2e-5


@pytest.mark.parametrize("m,k,n", [(200, 1024, 512), (300, 4096, 1024), (64, 768, 768)])
def test_linear_output_type_the_dense_kernel_does_not_write(ops, m, k, n):
    # bf16 activations with an fp16 result: the in-pipeline kernel, split or not, whatever the model prefers
    packed, books, w = _weight(ops, n, k, 4, torch.float16, seed=m)
    x, bias = torch.randn(m, k, device="cuda").bfloat16(), torch.randn(n, device="cuda")
    y = ops.dimq_linear_wq(x, packed, books, bias, n, k, bits=4, out_dtype=torch.float16)
    assert y.dtype == torch.float16 and ops.last_device_status() == 0
    assert _rel(y, x.double() @ w.t() + bias.double()) < 2.0 ** -12 + 1.2e-5


@pytest.mark.parametrize("n", [100, 500, 1004])
@pytest.mark.parametrize("m,k", [(33, 1024), (64, 4096), (197, 1024), (512, 2048), (1000, 4096), (1025, 2048), (2000, 1024)])
def test_linear_fp32_result_in_rows_the_16_bit_form_cannot_write(ops, m, k, n):
    # N % 8 == 4: the split or unsplit in-pipeline kernel, with the scratch its query reports
    packed, books, w = _weight(ops, n, k, 4, torch.float16, seed=m)
    x, bias = torch.randn(m, k, device="cuda").bfloat16(), torch.randn(n, device="cuda")
    y = ops.dimq_linear_wq(x, packed, books, bias, n, k, bits=4)
    assert y.dtype == torch.float32 and ops.last_device_status() == 0
    # hi + lo codewords carry 2^-17; the accumulators truncate, 1.2e-6 per 1024 products
    assert _rel(y, x.double() @ w.t() + bias.double()) < 1.2e-5


@pytest.mark.parametrize("m,k,n", [(384, 4096, 1024), (384, 8192, 512), (197, 1024, 1024), (197, 2048, 1000), (576, 4096, 512)])
@pytest.mark.parametrize("act,book", [(torch.float16, torch.float16), (torch.bfloat16, torch.bfloat16),
                                      (torch.bfloat16, torch.float16)])
def test_linear_fp32_result_below_1024_rows_sums_in_slices(ops, m, k, n, act, book):
    # The tensor cores' accumulators lose 1.25e-9 of a sum per product (6.4e-7 at 512, 3.7e-6 at 3072).  These shapes are cut
    # into at least four slices of K; where bf16 activations meet fp16 codewords each product is a hi + lo pair.
    packed, books, w = _weight(ops, n, k, 4, book, seed=m)
    x = torch.randn(m, k, device="cuda").to(act)
    y = ops.dimq_linear_wq(x, packed, books, None, n, k, bits=4)
    assert y.dtype == torch.float32 and ops.last_device_status() == 0
    assert _rel(y, x.double() @ w.t()) < 1.1 * 1.25e-9 * k / 4 * (1 if act == book else 2)


@pytest.mark.parametrize("act,out,kernels", [(torch.float32, torch.float32, 2), (torch.float32, torch.bfloat16, 1),
                                             (torch.bfloat16, torch.float16, 1), (torch.bfloat16, torch.float32, 2)])
def test_linear_scratch_and_launch_count_follow_the_output(ops, act, out, kernels):
    from dimq_b200 import _lib

    m, k, n = 2000, 1024, 512
    packed, books, w = _weight(ops, n, k, 4, torch.float16, seed=3)
    x = torch.randn(m, k, device="cuda").to(act)
    ops.dimq_linear_wq(x, packed, books, None, n, k, bits=4, out_dtype=out)
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    before, count = torch.cuda.memory_allocated(), _lib.LAUNCH_COUNT[0]
    y = ops.dimq_linear_wq(x, packed, books, None, n, k, bits=4, out_dtype=out)
    assert _lib.LAUNCH_COUNT[0] - count == kernels
    extra = torch.cuda.max_memory_allocated() - before - y.numel() * y.element_size()
    if act == torch.float32:
        assert (extra > 4 * m * k) == (out == torch.float32)     # the split activations, where they are used
    assert _rel(y, x.double() @ w.t()) < {torch.float32: 1.2e-5, torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11}[out]


@pytest.mark.parametrize("out,kernels", [(torch.bfloat16, 2), (torch.float32, 2), (torch.float16, 1)])
def test_conv_launch_count_follows_the_output(ops, out, kernels):
    from dimq_b200 import _lib

    packed, books, w = _weight(ops, 64, 64, 4, torch.bfloat16, seed=4)
    x = torch.randn(4, 64, 20, 20, device="cuda").bfloat16().contiguous(memory_format=torch.channels_last)
    khwc = ops.conv_prepack(packed, (64, 64, 1, 1), 4)
    count = _lib.LAUNCH_COUNT[0]
    y = ops.dimq_conv2d_wq(x, packed, books.reshape(-1), None, (64, 64, 1, 1), bits=4, out_dtype=out, packed_khwc=khwc)
    assert _lib.LAUNCH_COUNT[0] - count == kernels
    want = F.conv2d(x.double().contiguous(), w.view(64, 64, 1, 1))
    assert _rel(y, want) < {torch.float32: 1.2e-5, torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11}[out]


def test_a4_row_limit_is_the_one_ops_states(ops, monkeypatch):
    # rows of 3 fp32 elements: not the fp32-grade form; the limit chooses between the bf16 pair (two launches) and the table
    from dimq_b200 import _lib

    m, k, n = 600, 128, 3
    packed, books, w = _weight(ops, n, k, 4, torch.float32, seed=8)
    x = torch.randn(m, k, device="cuda")
    want = _codes(x, 0.23, 7) @ w.t()
    for limit, kernels in ((ops.A4_TC_MIN_ROWS, 2), (m, 2), (m + 1, 1)):
        monkeypatch.setattr(ops, "A4_TC_MIN_ROWS", limit)
        count = _lib.LAUNCH_COUNT[0]
        y = ops.dimq_linear_lut(x, packed, books.reshape(-1), 0.23, 7, None, n, k)
        assert _lib.LAUNCH_COUNT[0] - count == kernels, limit
        assert _rel(y, want) < 1.2e-5


def test_operands_on_another_device_are_refused(ops):
    # the host path hands raw pointers to the kernels: each operand is checked before any launch
    m, k, n = 64, 128, 64
    packed, books, _ = _weight(ops, n, k, 4, torch.float16, seed=2)
    x, bias, res = torch.randn(m, k, device="cuda"), torch.randn(n, device="cuda"), torch.randn(m, n, device="cuda")
    img = torch.randn(2, 64, 8, 8, device="cuda")
    cp, cb, _ = _weight(ops, 64, 64, 4, torch.float16, seed=3)
    cb = cb.reshape(-1)
    conv = (None, (64, 64, 1, 1))
    h = torch.randn(4, 128, device="cuda").bfloat16()
    g = torch.ones(128, device="cuda")
    calls = [
        lambda: ops.dimq_linear_wq(x, packed, books, bias, n, k, residual=res.cpu()),
        lambda: ops.dimq_linear_wq(x, packed, books, bias.cpu(), n, k),
        lambda: ops.dimq_linear_wq(x, packed.cpu(), books, bias, n, k),
        lambda: ops.dimq_linear_wq(x, packed, books.cpu(), bias, n, k),
        lambda: ops.dimq_linear_wq(x, packed, books, bias, n, k, packed_tiled=packed.cpu()),
        lambda: ops.dimq_linear_a4(x, packed, books.reshape(-1), 0.1, 3, None, n, k, residual=res.cpu()),
        lambda: ops.dimq_conv2d_wq(img, cp, cb, *conv, residual=torch.zeros(2, 64, 8, 8)),
        lambda: ops.dimq_conv2d_wq(img, cp, cb, *conv, packed_khwc=cp.cpu()),
        lambda: ops.add_layer_norm(h, h.cpu(), g, g),
        lambda: ops.add_layer_norm(h, None, g.cpu(), g),
        lambda: ops.add_layer_norm(h, None, g, g.cpu()),
    ]
    for i, call in enumerate(calls):
        with pytest.raises(RuntimeError, match="device|CUDA"):
            call()
            torch.cuda.synchronize()
            raise AssertionError(f"call {i} was accepted")


@pytest.mark.parametrize("act,book,bound", [(torch.float32, torch.float32, 4 * REL), (torch.float32, torch.float16, 4 * REL),
                                            (torch.float32, torch.bfloat16, 4 * REL), (torch.bfloat16, torch.float16, 1.2e-5)])
def test_linear_rows_of_every_size(ops, act, book, bound):
    # rows from the subnormals to 1e33 (both forms scale a row by a power of two into fp16's range), each against its own norm
    m, k, n = 1100, 768, 64
    packed, books, w = _weight(ops, n, k, 4, book, seed=17)
    books, w = books * 64, w * 64                                # about 1
    size = 10.0 ** torch.linspace(-36.5, 33, m, device="cuda", dtype=torch.float64).view(-1, 1)
    x = (torch.randn(m, k, device="cuda", dtype=torch.float64) * size).to(act)
    y = ops.dimq_linear_wq(x, packed, books, None, n, k, bits=4)
    assert y.dtype == torch.float32 and ops.last_device_status() == 0
    err = (y.double() - x.double() @ w.t()).norm(dim=1) / (x.double().norm(dim=1) * w.norm() / k ** 0.5)
    assert float(err.max()) < bound


@pytest.mark.parametrize("xs,ws", [(1e-42, 1e12), (1e-30, 1e30), (1e30, 1e-30), (1e12, 1e-42), (1e-20, 1e-16), (1e20, 1e14), (1e-36, 1e36)])
def test_linear_f32_scales_that_meet(ops, xs, ws):
    # rows and codewords of opposite extremes: the scales are undone one after the other
    m, k, n = 130, 768, 64
    packed, books, w = _weight(ops, n, k, 4, torch.float32, seed=18)
    books = (books.double() * 50 * ws).float()
    idx = torch.stack([packed.view(n, -1) & 15, packed.view(n, -1) >> 4], 2).view(n, k).long()
    w = books.double().reshape(-1)[idx]
    x = (torch.randn(m, k, device="cuda", dtype=torch.float64) * xs).float()
    y = ops.dimq_linear_wq(x, packed, books, None, n, k, bits=4)
    assert _rel(y, x.double() @ w.t()) < 4 * REL


@pytest.mark.parametrize("m,k,n", [(40, 64, 64), (300, 192, 132), (197, 768, 1000), (130, 1088, 64)])
@pytest.mark.parametrize("book", [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("outlier", [1.0, 1e5, 1e8])
def test_linear_f32_rows_with_an_outlier(ops, m, k, n, book, outlier):
    # one activation per row far above the others, which meets zero codewords; K of odd and even numbers of 64
    packed, books, w = _weight(ops, n, k, 4, book, seed=m)
    idx = torch.stack([packed.view(n, -1) & 15, packed.view(n, -1) >> 4], 2).view(n, k)
    idx[:, 5] = 3
    books = books.reshape(-1).clone()
    books[3] = 0
    packed, w = ops.pack_bits(idx, 4), books.double()[idx.long()]
    x = torch.randn(m, k, device="cuda")
    x[:, 5] = outlier * x[:, 5].sign()
    y = ops.dimq_linear_wq(x, packed, books, None, n, k, bits=4)
    assert ops.last_device_status() == 0 and _rel(y, x.double() @ w.t()) < REL


@pytest.mark.parametrize("k", [64, 192, 768])
@pytest.mark.parametrize("a4", [False, True])
def test_fp32_codebooks_with_an_outlier(ops, k, a4):
    # one codeword far above the others, which meets zero activations
    m, n = 150, 64
    packed, books, w = _weight(ops, n, k, 4, torch.float32, seed=k)
    idx = torch.stack([packed.view(n, -1) & 15, packed.view(n, -1) >> 4], 2).view(n, k)
    idx[idx == 3] = 4
    idx[:, 7] = 3
    books = books.reshape(-1).clone()
    books[3] = 1e6                            # 2^25 times the others
    packed, w = ops.pack_bits(idx, 4), books.double()[idx.long()]
    x = torch.randn(m, k, device="cuda")
    x[:, 7] = 0
    if a4:
        y, want = ops.dimq_linear_lut(x, packed, books, 0.23, 7, None, n, k), _codes(x, 0.23, 7) @ w.t()
    else:
        y, want = ops.dimq_linear_wq(x, packed, books, None, n, k, bits=4), x.double() @ w.t()
    assert ops.last_device_status() == 0 and _rel(y, want) < REL


@pytest.mark.parametrize("book", [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("bits,group_rows", [(4, None), (3, 40), (2, 1)])
def test_linear_f32_non_finite_codewords(ops, book, bits, group_rows):
    # an infinite or NaN codeword gives what fp32 products and sums give, whatever its type
    m, k, n = 140, 192, 100
    packed, books, _ = _weight(ops, n, k, bits, book, group_rows, seed=6)
    books = books.clamp(-1e3, 1e3)
    books[0, 1], books[-1, 2] = float("inf"), float("-inf")
    if books.shape[0] > 2:
        books[1, 0] = float("nan")
    idx = ops.unpack_bits(packed, n * k, bits).view(n, k).long()
    idx[3:7], idx[9, ::2] = 3, 0                 # columns of finite codewords only, and a mixed one
    packed = ops.pack_bits(idx.to(torch.uint8), bits)
    rows = torch.arange(n, device="cuda") // (group_rows or n)
    w = torch.gather(books.float()[rows], 1, idx)
    x = torch.randn(m, k, device="cuda")
    x[5], x[6], x[:, 11] = 0.0, x[6].bfloat16().float(), x[:, 11].half().float()      # zeros, and values exact in one term
    x[7, 3], x[8, 4], x[9, 5] = float("inf"), float("-inf"), float("nan")
    x[10] *= torch.logspace(0, -30, k, device="cuda")
    y = ops.dimq_linear_wq(x, packed, books if group_rows else books.reshape(-1), None, n, k, bits=bits, group_rows=group_rows)
    # infinities and NaN of the sum follow from those of its products, in any order
    prod = x.unsqueeze(1) * w.unsqueeze(0)
    nan = prod.isnan().any(2) | ((prod == float("inf")).any(2) & (prod == float("-inf")).any(2))
    sign = (prod == float("inf")).any(2).float() - (prod == float("-inf")).any(2).float()
    assert torch.equal(y.isnan(), nan)
    assert torch.equal(y.isinf(), ~nan & (sign != 0)) and torch.equal(y[y.isinf()].sign(), sign[y.isinf()])
    ok = y.isfinite()
    want = torch.nan_to_num(x.double(), 0, 0, 0) @ torch.nan_to_num(w.double(), 0, 0, 0).t()
    bound = 1e-6 * torch.nan_to_num(x.double(), 0, 0, 0).norm(dim=1, keepdim=True) * torch.nan_to_num(w.double(), 0, 0, 0).norm(dim=1)
    assert bool(((y.double() - want).abs() <= bound + 1e-30)[ok].all())


@pytest.mark.parametrize("book", [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("bits", [2, 3, 4])
def test_linear_f32_infinite_activations_against_finite_codewords(ops, book, bits):
    # zero, subnormal, smallest and largest codewords of either sign: what the tensor cores give stands, NaN included
    m, k, n = 200, 192, 132
    packed, books, _ = _weight(ops, n, k, bits, book, seed=bits)
    books = books.reshape(-1).clone()
    f = torch.finfo(book)
    books[0], books[1] = 0.0, -f.smallest_normal / 64
    if bits > 2:
        books[2], books[3] = f.smallest_normal, -f.max / 64      # no product of a finite activation overflows
    idx = ops.unpack_bits(packed, n * k, bits).view(n, k).long()
    idx[5:9] = books.numel() - 1                  # columns without a zero codeword
    packed, w = ops.pack_bits(idx.to(torch.uint8), bits), books.float()[idx]
    x = torch.randn(m, k, device="cuda")
    x[3, 5], x[40, 9], x[199, 191] = float("inf"), float("-inf"), float("inf")
    x[50, 1], x[50, 2], x[60, 0] = float("inf"), float("-inf"), float("nan")
    y = ops.dimq_linear_wq(x, packed, books, None, n, k, bits=bits)
    assert ops.last_device_status() == 0
    rows = [3, 40, 50, 60, 199]
    prod = x[rows].unsqueeze(1) * w.unsqueeze(0)
    plus, minus = (prod == float("inf")).any(2), (prod == float("-inf")).any(2)
    nan = prod.isnan().any(2) | (plus & minus)
    assert torch.equal(y[rows].isnan(), nan)
    assert torch.equal(y[rows] == float("inf"), plus & ~nan) and torch.equal(y[rows] == float("-inf"), minus & ~nan)


def test_infinite_activations_cost_no_second_computation(ops):
    # Outputs are computed again only where the codebook has an infinity or a NaN (that took 40 times the time here).
    m, k, n = 1576, 768, 3072
    packed, books, _ = _weight(ops, n, k, 4, torch.float32, seed=1)
    books = books.reshape(-1).clone()
    books[2] = 0.0
    x = torch.randn(m, k, device="cuda")
    bad = x.clone()
    bad[:, 5] = float("inf")

    def us(act):
        start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        best = float("inf")
        for _ in range(5):
            start.record()
            for _ in range(3):
                ops.dimq_linear_wq(act, packed, books, None, n, k, bits=4)
            end.record()
            end.synchronize()
            best = min(best, start.elapsed_time(end))
        return best

    assert us(bad) < 3 * us(x)


def test_linear_f32_infinite_activations_against_tiny_codewords(ops):
    # a codeword far below the largest of its book is not zero: infinity times it is infinity
    m, k, n = 40, 64, 64
    books = torch.tensor([1e4, -1e4, 1e-20, -1e-20, 0.0] + [1.0] * 11, device="cuda")
    idx = torch.randint(5, 16, (n, k), device="cuda")
    idx[:, 0] = torch.arange(n, device="cuda") % 5
    x = torch.randn(m, k, device="cuda")
    x[3, 0], x[4, 0] = float("inf"), float("-inf")
    for book in (books, books.bfloat16()):
        y = ops.dimq_linear_wq(x, ops.pack_bits(idx.to(torch.uint8), 4), book, None, n, k, bits=4)
        want = x @ book.float()[idx].t()
        assert torch.equal(y.isnan(), want.isnan()) and torch.equal(y.isinf(), want.isinf())
        assert torch.equal(y[y.isinf()].sign(), want[want.isinf()].sign())
        assert _rel(y[:3], (x.double() @ book.double()[idx].t())[:3]) < REL
