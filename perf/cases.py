"""The work a user has this framework do, as cases that can be timed and compared.

A case is a dict of plain values.  ``listed()`` names twelve of them, ``draw(rng)`` gives more of the same
ranges, ``prepare(case, seed)`` makes what a program holds before the call (inputs, packed weights, the
module or model that owns them), ``run(state)`` is one pass through the public entry points, ``work(case)``
the bytes and operations a pass cannot do without, ``tolerance(case)`` how far two correct implementations
may lie apart, ``exact(case, seed)`` the outputs in 64 bits by plain torch.

Kinds:

* ``linear``: a weight-only ``DIMQLinear`` on 16-bit activations (2-, 3- or 4-bit indices), from one row
  (decode) over a few dozen (a small batch) to thousands (prefill, a batch of token sequences).
* ``linear_f32``: the same layer on fp32 activations and with an fp32 result.
* ``conv``: a weight-only ``DIMQConv2d`` on 16-bit channels_last activations.
* ``vit`` / ``resnet``: the whole-model forwards of ``dimq_b200.workloads``.
* ``linear_a4`` / ``conv_a4``: the W4A4 layers of a checkpoint of the reference: fp32 activations as
  PyTorch stores them (NCHW for the convolution), 4-bit activation codes, fp32 results.
* ``export``: nearest-codeword assignment and packing of a weight, and unpacking of what was packed.
* ``qat``: the straight-through fake quantisation of a training step, forward and backward.
"""

from __future__ import annotations

import math

import torch
import torch.nn.functional as F

from dimq_b200 import ops
from dimq_b200.export import activation_qparams_from_minmax
from dimq_b200.modules import DIMQConv2d, DIMQLinear
from dimq_b200.qat import fake_quant_weight
from dimq_b200.workloads import (VIT_B16, DIMQResNet18, DIMQViT, build_resnet18_checkpoint, build_vit_b16_checkpoint,
                                 quantile_codebooks)

_DTYPES = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}


def listed() -> list[dict]:
    return [
        # one token through a ViT-L MLP layer: the smallest call, all launch and host latency
        dict(name="decode_m1", kind="linear", m=1, k=1024, n=4096, bits=4, group_rows=0, act="bf16", book="f16",
             epilogue="gelu"),
        # eight sequences decoding against a large square weight: 32 MB of indices to stream
        dict(name="decode_m8_large", kind="linear", m=8, k=8192, n=8192, bits=4, group_rows=0, act="bf16", book="f16",
             epilogue="none"),
        # a small batch of rows through the other ViT-L MLP layer: long K, few output tiles
        dict(name="linear_m64", kind="linear", m=64, k=4096, n=1024, bits=2, group_rows=128, act="bf16", book="bf16",
             epilogue="none"),
        # eight images of 197 tokens, fp32 end to end, the reference export's fp16 16-entry codebook per layer
        dict(name="linear_f32_m1576", kind="linear_f32", m=1576, k=768, n=3072, bits=4, group_rows=0, book="f32"),
        # one ResNet basic-block convolution with a codebook per output channel
        dict(name="conv_64ch_b64", kind="conv", batch=64, cin=64, cout=64, size=56, ksize=3, stride=1, bits=4,
             group_rows=1, act="bf16", book="f16", epilogue="relu"),
        # whole-model throughput: ResNet-18, 4-bit layers, 8-bit stem and classifier
        dict(name="resnet18_b256", kind="resnet", batch=256),
        # whole-model throughput: ViT-B/16, 3-bit layers with a codebook per 128 rows
        dict(name="vit_b16_b128", kind="vit", batch=128),
        # whole-model latency: one image
        dict(name="vit_b16_b1", kind="vit", batch=1),
        # a W4A4 layer of an exported checkpoint on the tokens of one image
        dict(name="linear_a4_m197", kind="linear_a4", m=197, k=768, n=3072, book="f16"),
        # a W4A4 convolution of an exported checkpoint on a small batch of NCHW feature maps
        dict(name="conv_a4_nchw_b7", kind="conv_a4", batch=7, cin=128, cout=128, size=28, ksize=3, stride=1, book="f16"),
        # export of one layer: assign, pack, and unpack as a loader does
        dict(name="export_4096x1024", kind="export", n=4096, k=1024, bits=4, group_rows=0),
        # one layer's share of a QAT step: the 512-channel 3x3 convolution weight
        dict(name="qat_512ch", kind="qat", n=512, k=512 * 9, bits=4, group_rows=0),
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng) -> dict:
    kind = rng.choice(["linear", "linear", "linear", "linear_f32", "conv", "resnet", "vit", "linear_a4", "conv_a4",
                       "export", "qat"])
    if kind == "linear":
        k = rng.choice([512, 768, 1024, 3072, 4096, 8192])
        n = rng.choice([768, 1000, 1024, 2304, 3072, 4096, 8192])
        return dict(kind=kind, m=_log_int(rng, 1, 8192), k=k, n=n, bits=rng.choice([2, 3, 4]),
                    group_rows=rng.choice([0, 128]), act=rng.choice(["bf16", "bf16", "f16"]),
                    book=rng.choice(["f16", "bf16"]), epilogue=rng.choice(["none", "gelu"]))
    if kind == "linear_f32":
        return dict(kind=kind, m=_log_int(rng, 1, 4096), k=rng.choice([512, 768, 1024, 3072]),
                    n=rng.choice([768, 1000, 2304, 3072]), bits=rng.choice([2, 3, 4]), group_rows=rng.choice([0, 128]),
                    book=rng.choice(["f32", "f16"]))
    if kind == "conv":
        cin, size = rng.choice([(64, 56), (128, 28), (256, 14), (512, 7)])
        stride = rng.choice([1, 1, 2])
        return dict(kind=kind, batch=_log_int(rng, 1, 128), cin=cin, cout=cin * stride, size=size,
                    ksize=rng.choice([1, 3, 3, 3]), stride=stride, bits=rng.choice([2, 4]), group_rows=rng.choice([0, 1]),
                    act=rng.choice(["bf16", "f16"]), book=rng.choice(["f16", "bf16"]),
                    epilogue=rng.choice(["none", "relu"]))
    if kind == "resnet":
        return dict(kind=kind, batch=_log_int(rng, 1, 256))
    if kind == "vit":
        return dict(kind=kind, batch=_log_int(rng, 1, 128))
    if kind == "linear_a4":
        return dict(kind=kind, m=_log_int(rng, 1, 4096), k=rng.choice([512, 768, 1024, 3072]),
                    n=rng.choice([768, 1000, 2304, 3072]), book=rng.choice(["f16", "f16", "f32"]))
    if kind == "conv_a4":
        cin, size = rng.choice([(64, 56), (128, 28), (256, 14), (512, 7)])
        stride = rng.choice([1, 1, 2])
        return dict(kind=kind, batch=_log_int(rng, 1, 64), cin=cin, cout=cin * stride, size=size,
                    ksize=rng.choice([1, 3, 3]), stride=stride, book=rng.choice(["f16", "f16", "f32"]))
    if kind == "export":
        return dict(kind=kind, n=_log_int(rng, 64, 8192), k=rng.choice([147, 512, 576, 1024, 4608]),
                    bits=rng.choice([2, 3, 4, 8]), group_rows=rng.choice([0, 0, 128]))
    return dict(kind=kind, n=_log_int(rng, 64, 8192), k=rng.choice([147, 512, 576, 1024, 4608]),
                bits=rng.choice([2, 3, 4, 8]), group_rows=rng.choice([0, 0, 128]))


# ---------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------

def _codebooks(w: torch.Tensor, entries: int, group_rows: int) -> torch.Tensor:
    """Quantile codebooks ``[G, entries]`` (fp32) from at most a few thousand columns of every row."""
    rows = w.shape[0]
    columns = max(1, min(w.shape[1], (1 << 22) // rows))
    return quantile_codebooks(w[:, :columns], entries, group_rows)


def _packed_weight(n: int, k: int, bits: int, group_rows: int, book: str, gen, std: float = 0.02):
    """N(0, std) weight -> quantile codebook(s), stored in ``book`` -> nearest-codeword indices, packed."""
    w = torch.randn(n, k, device="cuda", generator=gen) * std
    rows = group_rows or n
    books = _codebooks(w, 1 << bits, rows).to(_DTYPES[book])
    _, packed = ops.hard_quantize(w, books.float(), group_rows=rows, bits=bits, return_indices=False)
    return packed, books


def prepare(case: dict, seed: int):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind = case["kind"]
    if kind in ("linear", "linear_f32"):
        act = case.get("act", "f32")
        m, k, n = case["m"], case["k"], case["n"]
        packed, books = _packed_weight(n, k, case["bits"], case["group_rows"], case["book"], gen)
        bias = torch.randn(n, device="cuda", generator=gen).mul_(0.02).to(_DTYPES[act])
        epilogue = case.get("epilogue", "none")
        layer = DIMQLinear(packed, books, None, None, n, k, bias, bits=case["bits"],
                           group_rows=case["group_rows"] or None, out_dtype=_DTYPES[act],
                           epilogue=None if epilogue == "none" else epilogue)
        x = torch.randn(m, k, device="cuda", generator=gen).to(_DTYPES[act])
        return layer, x
    if kind == "conv":
        cin, cout, ks = case["cin"], case["cout"], case["ksize"]
        packed, books = _packed_weight(cout, cin * ks * ks, case["bits"], case["group_rows"], case["book"], gen,
                                       std=(2.0 / (cin * ks * ks)) ** 0.5)
        bias = torch.randn(cout, device="cuda", generator=gen).mul_(0.1).to(_DTYPES[case["act"]])
        layer = DIMQConv2d(packed, books, None, None, (cout, cin, ks, ks), bias, stride=case["stride"],
                           padding=ks // 2, bits=case["bits"], group_rows=case["group_rows"] or None,
                           out_dtype=_DTYPES[case["act"]],
                           epilogue=None if case["epilogue"] == "none" else case["epilogue"])
        x = torch.randn(case["batch"], cin, case["size"], case["size"], device="cuda", generator=gen).relu_()
        return layer, x.to(_DTYPES[case["act"]]).contiguous(memory_format=torch.channels_last)
    if kind == "linear_a4":
        m, k, n = case["m"], case["k"], case["n"]
        packed, books = _packed_weight(n, k, 4, 0, case["book"], gen)
        bias = torch.randn(n, device="cuda", generator=gen).mul_(0.02)
        q = activation_qparams_from_minmax(-3.7, 3.9)
        layer = DIMQLinear(packed, books.reshape(-1), q["scale"], q["zero_point"], n, k, bias)
        return layer, torch.randn(m, k, device="cuda", generator=gen)
    if kind == "conv_a4":
        cin, cout, ks = case["cin"], case["cout"], case["ksize"]
        packed, books = _packed_weight(cout, cin * ks * ks, 4, 0, case["book"], gen, std=(2.0 / (cin * ks * ks)) ** 0.5)
        bias = torch.randn(cout, device="cuda", generator=gen).mul_(0.1)
        q = activation_qparams_from_minmax(0.0, 4.2)
        layer = DIMQConv2d(packed, books.reshape(-1), q["scale"], q["zero_point"], (cout, cin, ks, ks), bias,
                           stride=case["stride"], padding=ks // 2)
        return layer, torch.randn(case["batch"], cin, case["size"], case["size"], device="cuda", generator=gen).relu_()
    if kind == "resnet":
        model = DIMQResNet18(build_resnet18_checkpoint(seed=seed)).eval()
        return model, torch.randn(case["batch"], 3, 224, 224, device="cuda", generator=gen)
    if kind == "vit":
        model = DIMQViT(build_vit_b16_checkpoint(seed=seed)).eval()
        return model, torch.randn(case["batch"], 3, 224, 224, device="cuda", generator=gen)
    w = torch.randn(case["n"], case["k"], device="cuda", generator=gen) * 0.02
    rows = case["group_rows"] or case["n"]
    books = _codebooks(w, 1 << case["bits"], rows)
    if rows == case["n"]:
        books = books.reshape(-1)
    if kind == "export":
        return w, books, case["group_rows"] or None, case["bits"]
    grad = torch.randn(case["n"], case["k"], device="cuda", generator=gen) * 1e-3
    return w.requires_grad_(True), books, case["group_rows"] or None, grad


# ---------------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------------

def run(state):
    if len(state) == 2:                         # a layer or a model, and its input
        module, x = state
        with torch.no_grad():
            return module(x)
    if isinstance(state[3], int):               # export
        w, books, group_rows, bits = state
        indices, packed = ops.hard_quantize(w, books, group_rows=group_rows, bits=bits)
        return indices, packed, ops.unpack_bits(packed, w.numel(), bits)
    w, books, group_rows, grad = state          # quantisation-aware training
    w.grad = None
    out = fake_quant_weight(w, books, group_rows=group_rows)
    out.backward(grad)
    return out.detach(), w.grad


# ---------------------------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------------------------

def _unpack64(packed: torch.Tensor, numel: int, bits: int) -> torch.Tensor:
    """Indices of a little-endian bit stream, with plain torch."""
    stream = (packed.view(-1, 1) >> torch.arange(8, device=packed.device, dtype=torch.uint8)) & 1
    fields = stream.view(-1)[:numel * bits].view(numel, bits).long()
    return (fields << torch.arange(bits, device=packed.device)).sum(1)


def _weight64(packed: torch.Tensor, books: torch.Tensor, n: int, k: int, bits: int, group_rows: int) -> torch.Tensor:
    idx = _unpack64(packed, n * k, bits).view(n, k)
    books = books.double().reshape(-1, books.shape[-1])
    rows = books[torch.arange(n, device=idx.device) // (group_rows or n)]        # [n, entries]
    return torch.gather(rows, 1, idx)


def _layer64(layer: dict) -> tuple[torch.Tensor, torch.Tensor]:
    """Weight (in its own shape) and bias of a checkpoint's layer."""
    shape = layer["weight_shape"]
    w = _weight64(layer["packed_weight"], layer["codebook"], shape[0], math.prod(shape[1:]), layer["bit_w"],
                  layer.get("group_rows") or 0)
    return w.view(*shape), layer["bias"].double()


def _centred64(x: torch.Tensor, q: dict) -> torch.Tensor:
    """4-bit activation codes without the zero point, times the scale (the quotient is an fp32 one by contract)."""
    scale = torch.tensor(q["scale"], device=x.device, dtype=torch.float32)
    z = q["zero_point"]
    return ((torch.round(x / scale) + z).clamp_(0, 15) - z).double() * scale.double()


def _resnet64(ckpt: dict, images: torch.Tensor) -> torch.Tensor:
    layers = {name: _layer64(layer) for name, layer in ckpt["layers"].items()}

    def conv(name, x):
        layer = ckpt["layers"][name]
        w, b = layers[name]
        return F.conv2d(x, w, b, layer["stride"], layer["padding"])

    logits = []
    for part in images.double().split(16):
        x = F.max_pool2d(conv("conv1", part).relu_(), 3, 2, 1)
        for stage in range(1, 5):
            for block in range(2):
                pre = f"layer{stage}.{block}."
                skip = conv(pre + "downsample", x) if pre + "downsample" in layers else x
                x = (conv(pre + "conv2", conv(pre + "conv1", x).relu_()) + skip).relu_()
        logits.append(F.linear(x.mean(dim=(2, 3)), *layers["fc"]))
    return torch.cat(logits)


def _vit64(ckpt: dict, images: torch.Tensor) -> torch.Tensor:
    cfg = ckpt["config"]
    hid, heads = cfg["hidden"], cfg["heads"]
    layers = {name: _layer64(layer) for name, layer in ckpt["layers"].items()}
    dense = {name: value.double() for name, value in ckpt["non_quantized_state_dict"].items()}

    def norm(name, x):
        return F.layer_norm(x, (hid,), dense[name + ".weight"], dense[name + ".bias"], 1e-6)

    logits = []
    for part in images.double().split(16):
        patches = F.conv2d(part, dense["patch_embed.weight"], dense["patch_embed.bias"], stride=cfg["patch"])
        b = part.shape[0]
        x = torch.cat([dense["cls_token"].expand(b, 1, hid), patches.flatten(2).transpose(1, 2)], 1) + dense["pos_embed"]
        for i in range(cfg["layers"]):
            pre = f"blocks.{i}."
            qkv = F.linear(norm(pre + "norm1", x), *layers[pre + "attn.qkv"])
            q, k, v = qkv.view(b, -1, 3, heads, hid // heads).permute(2, 0, 3, 1, 4)
            a = torch.softmax(q @ k.transpose(-1, -2) * (hid // heads) ** -0.5, -1) @ v
            x = x + F.linear(a.transpose(1, 2).reshape(b, -1, hid), *layers[pre + "attn.proj"])
            h = F.gelu(F.linear(norm(pre + "norm2", x), *layers[pre + "mlp.fc1"]))
            x = x + F.linear(h, *layers[pre + "mlp.fc2"])
        logits.append(F.linear(norm("norm", x[:, 0]), *layers["head"]))
    return torch.cat(logits)


def exact(case: dict, seed: int):
    """What ``run`` returns for the inputs of ``prepare(case, seed)``, in 64 bits and with plain torch."""
    kind = case["kind"]
    if kind in ("resnet", "vit"):
        gen = torch.Generator(device="cuda").manual_seed(seed)
        images = torch.randn(case["batch"], 3, 224, 224, device="cuda", generator=gen)
        if kind == "resnet":
            return _resnet64(build_resnet18_checkpoint(seed=seed), images)
        return _vit64(build_vit_b16_checkpoint(seed=seed), images)
    if kind == "export":
        return None                                # whole numbers and bytes
    if kind == "qat":
        w, books, _, grad = prepare(case, seed)
        w = w.detach().double()
        books = books.double().reshape(-1, books.shape[-1]).sort(dim=1).values
        rows = case["group_rows"] or case["n"]
        out = torch.empty_like(w)
        for g, book in enumerate(books):
            part = w[g * rows:(g + 1) * rows]
            out[g * rows:(g + 1) * rows] = book[torch.bucketize(part, (book[1:] + book[:-1]) / 2)]
        return out, grad.double()
    layer, x = prepare(case, seed)
    bits = case.get("bits", 4)
    n = case["cout"] if "cout" in case else case["n"]
    ks = case.get("ksize", 1)
    k = case["cin"] * ks * ks if "cout" in case else case["k"]
    w = _weight64(layer.packed_weight, layer.codebook, n, k, bits, case.get("group_rows", 0))
    if kind == "linear_a4":
        x = _centred64(x, activation_qparams_from_minmax(-3.7, 3.9))
    elif kind == "conv_a4":
        x = _centred64(x, activation_qparams_from_minmax(0.0, 4.2))
    x, bias = x.double(), layer.bias.double()
    if "cout" in case:
        y = torch.cat([F.conv2d(part.contiguous(), w.view(n, case["cin"], ks, ks), bias, case["stride"], ks // 2)
                       for part in x.split(16)])
    else:
        y = F.linear(x, w, bias)
    epilogue = case.get("epilogue", "none")
    return y.relu_() if epilogue == "relu" else F.gelu(y) if epilogue == "gelu" else y


# ---------------------------------------------------------------------------------------------
# what a pass cannot do without, and how exact it is
# ---------------------------------------------------------------------------------------------

def work(case: dict) -> dict:
    kind = case["kind"]
    size = {"f32": 4, "f16": 2, "bf16": 2}
    if kind in ("linear", "linear_f32", "linear_a4"):
        m, k, n = case["m"], case["k"], case["n"]
        io = size[case.get("act", "f32")]
        return {"bytes": m * k * io + m * n * io + n * k * case.get("bits", 4) / 8, "flops": 2.0 * m * n * k}
    if kind in ("conv", "conv_a4"):
        b, cin, cout, ks = case["batch"], case["cin"], case["cout"], case["ksize"]
        out = (case["size"] + 2 * (ks // 2) - ks) // case["stride"] + 1
        io = size[case.get("act", "f32")]
        weights = cout * cin * ks * ks
        return {"bytes": io * b * (cin * case["size"] ** 2 + cout * out * out) + weights * case.get("bits", 4) / 8,
                "flops": 2.0 * b * out * out * weights}
    if kind == "resnet":
        # images in, logits out, weights once; the layers' products (1.81 GMAC per image with the shortcuts)
        return {"bytes": case["batch"] * (3 * 224 * 224 * 4 + 4000) + 11.2e6 / 2,
                "flops": 928.8e9 / 256 * case["batch"]}
    if kind == "vit":
        cfg, t = VIT_B16, 197
        hid = cfg["hidden"]
        linears = cfg["layers"] * (4 * hid * hid + 2 * hid * cfg["mlp"])
        per_image = 2.0 * (t * linears + cfg["layers"] * 2 * t * t * hid + (t - 1) * hid * hid + hid * cfg["classes"])
        return {"bytes": case["batch"] * (3 * 224 * 224 * 4 + 4000) + (linears + hid * cfg["classes"]) * 3 / 8
                + hid * hid * 2, "flops": per_image * case["batch"]}
    numel = case["n"] * case["k"]
    if kind == "export":
        # weight in, indices out, packed out and read back, unpacked indices out
        return {"bytes": numel * (4 + 1 + 2 * case["bits"] / 8 + 1), "flops": 0}
    # weight in, quantised weight out, gradient in, weight gradient out
    return {"bytes": numel * 4 * 4, "flops": 0}


def tolerance(case: dict):
    kind = case["kind"]
    if kind in ("export", "qat"):
        return "exact"
    if kind in ("linear_f32", "linear_a4", "conv_a4"):
        return {"rel": 1e-5}          # sums of fp32 products in another order
    if kind in ("linear", "conv"):
        # the 16-bit rounding of the result: 2^-9 / sqrt(3) of a bf16 value, 2^-12 / sqrt(3) of an fp16 one
        return {"rel": 7e-3 if case["act"] == "bf16" else 1e-3}
    return {"rel": 4e-2 if kind == "vit" else 1e-2}   # bf16 activations stored after every layer
