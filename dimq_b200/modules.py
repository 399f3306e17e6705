"""Runtime modules for packed DIMQ layers — drop-ins for ``dimq_backend.modules``.

Constructor and ``from_export_layer`` signatures follow
dimq_cuda_backend/dimq_backend/modules.py:14-150.  Differences, all additive:

* ``act_scale=None`` selects the weight-only mode (activations stay in floating
  point; ``y = x @ codebook[idx].T + bias``) instead of the W4A4 product-table mode;
* ``bits`` / ``group_rows`` describe 2-, 3-, 4- or 8-bit indices and one codebook per
  ``group_rows`` output rows (``codebook`` is then ``[G, K]``);
* ``out_dtype`` / ``epilogue`` choose the output type and a fused ReLU / GELU.

There is no Python fallback: inputs must be CUDA tensors and the compiled library
must be present, otherwise ``forward`` raises.
"""

from __future__ import annotations

from typing import Any, Mapping

import torch
import torch.nn as nn

from . import _lib, ops


def _eager(x: torch.Tensor, codebook: torch.Tensor, bias: torch.Tensor | None) -> bool:
    """Plain eager execution: no tracer, dispatch or function mode, tensor subclass, function transform or gradient that
    has to see the registered operator."""
    if not (type(x) is torch.Tensor and torch._C._len_torch_dispatch_stack() == 0
            and torch._C._len_torch_function_stack() == 0 and not torch._C._is_tracing()
            and torch._C._functorch.peek_interpreter_stack() is None):
        return False
    return not torch.is_grad_enabled() or not (x.requires_grad or codebook.requires_grad
                                               or (bias is not None and bias.requires_grad))


class _Derived:
    """A tensor derived from a module's buffer on the GPU, with what a later call needs to know before it may read it: that
    the buffer still is what it was, and that the writing of the tensor - on the stream of the call that first needed it -
    comes before.  Holds the buffer's storage, so that a new one cannot turn up at its address."""

    __slots__ = ("source", "address", "version", "extra", "value", "device", "event", "written", "builder", "streams")

    def __init__(self, source: torch.Tensor, extra, value: torch.Tensor) -> None:
        self.source, self.address, self.version = source.detach(), source.data_ptr(), source._version
        self.extra, self.value = extra, value
        self.device = value.get_device()
        self.event = _lib.host().record_event(self.device)
        self.written = False                     # known to be complete, for every stream
        self.builder = torch._C._cuda_getCurrentRawStream(self.device)
        self.streams = {self.builder}            # those the allocator knows to read the value

    def __reduce__(self):                        # copied and saved modules derive their own
        return type(None), ()

    def is_of(self, source: torch.Tensor, extra) -> bool:
        return self.address == source.data_ptr() and self.version == source._version and self.extra == extra

    def readable(self) -> bool:
        """Make the current stream wait for the value where it has to.  False in a graph capture that began before the
        value was written: a replay would not wait."""
        raw = torch._C._cuda_getCurrentRawStream(self.device)
        if self.written and raw in self.streams:
            return True
        if not self.written:
            host = _lib.host()
            if host.event_done(self.event):
                self.written = True
            elif host.capturing(self.device):
                return False
            elif raw != self.builder:
                host.wait_event(self.event, self.device)
        if raw not in self.streams:
            self.value.record_stream(torch.cuda.current_stream(self.device))
            self.streams.add(raw)
        return True


def _pair(value) -> tuple[int, int]:
    if isinstance(value, int):
        return int(value), int(value)
    if len(value) != 2:
        raise ValueError(f"expected pair, got {value!r}")
    return int(value[0]), int(value[1])


class _PackedBase(nn.Module):
    def _init_common(self, packed_weight, codebook, act_scale, act_zero_point, bias, use_cuda_kernel, bits,
                     group_rows, out_dtype, epilogue):
        self.register_buffer("packed_weight", packed_weight.contiguous().to(torch.uint8))
        self.register_buffer("codebook", codebook.contiguous())
        self.register_buffer("bias", None if bias is None else bias.contiguous())
        self.act_scale = None if act_scale is None else float(act_scale)
        self.act_zero_point = int(act_zero_point) if act_zero_point is not None else 0
        self.use_cuda_kernel = bool(use_cuda_kernel)
        self.bits = int(bits)
        self.group_rows = None if group_rows is None else int(group_rows)
        self.out_dtype = out_dtype
        self.epilogue = epilogue
        if self.act_scale is not None and (self.bits != 4 or codebook.numel() != 16):
            raise ValueError("the W4A4 mode needs 4-bit indices and one 16-entry codebook; "
                             "pass act_scale=None for weight-only layers")

    def _kept(self, slot: str, source: torch.Tensor, extra=None) -> torch.Tensor | None:
        """What is kept in ``slot``, if ``source`` still is the buffer it was derived from and the current stream may read it."""
        kept = self.__dict__.get(slot)
        if type(kept) is _Derived and not source.is_inference() and kept.is_of(source, extra) and kept.readable():
            return kept.value
        return None

    def _keep(self, slot: str, source: torch.Tensor, value: torch.Tensor, extra=None) -> torch.Tensor:
        """Keep ``value``, just derived from the buffer ``source``, until that is replaced, moved or written in place.  Not
        kept: what a graph capture builds (only a replay writes it), and what an inference tensor gives (its writes are not
        counted)."""
        if not source.is_inference() and not _lib.host().capturing(value.get_device()):
            self.__dict__[slot] = _Derived(source, extra, value)
        return value

    def _apply(self, fn, recurse=True):
        super()._apply(fn, recurse)
        for slot, name in (("_tiled", "packed_weight"), ("_khwc", "packed_weight"), ("_scaled_cb", "codebook")):
            kept, source = self.__dict__.get(slot), getattr(self, name)
            if type(kept) is _Derived and (source.is_inference() or not kept.is_of(source, kept.extra)):
                self.__dict__[slot] = None           # a moved module leaves nothing behind
        return self

    def _scaled_codebook(self) -> torch.Tensor:
        """``act_scale * codebook`` in fp32 (the weight operand of the tensor-core W4A4 form), built once
        and rebuilt when the codebook buffer or the scale changes."""
        cb = self.codebook
        scaled = self._kept("_scaled_cb", cb, self.act_scale)
        if scaled is None:
            scale = torch.tensor(self.act_scale, dtype=torch.float32, device=cb.device)
            scaled = self._keep("_scaled_cb", cb, cb.detach().float().reshape(-1) * scale, self.act_scale)
        return scaled

    def _refuse(self) -> None:
        if not self.use_cuda_kernel:
            raise RuntimeError("dimq_b200 has no Python fallback path (use_cuda_kernel=False is not supported)")
        raise RuntimeError("dimq_b200 layers run on CUDA tensors only; move the module and its input to a B200")


class DIMQLinear(_PackedBase):
    """Linear layer backed by packed weight indices and a learned codebook."""

    def __init__(self, packed_weight, codebook, act_scale, act_zero_point, out_features, in_features, bias=None, *,
                 use_cuda_kernel: bool = True, bits: int = 4, group_rows: int | None = None,
                 out_dtype: torch.dtype | None = None, epilogue: str | None = None) -> None:
        super().__init__()
        self._init_common(packed_weight, codebook, act_scale, act_zero_point, bias, use_cuda_kernel, bits,
                          group_rows, out_dtype, epilogue)
        self.out_features = int(out_features)
        self.in_features = int(in_features)
        # indices re-ordered for the small-M kernel: built the first time a call with at most 16 activation
        # rows meets a weight that kernel takes (a second copy of the indices), rebuilt whenever the
        # packed_weight buffer is replaced, moved or written in place
        self._tiled = None

    def _prepacked(self, rows: int, x: torch.Tensor) -> torch.Tensor | None:
        if (rows > 16 or self.bits not in (2, 3, 4) or self.out_features % 16 != 0 or self.in_features % 128 != 0
                or self.in_features < 2048
                or x.dtype not in (torch.float16, torch.bfloat16)
                or self.out_features * self.in_features * self.bits < (1 << 24)):
            return None
        pw = self.packed_weight
        tiled = self._kept("_tiled", pw)
        if tiled is None:
            tiled = self._keep("_tiled", pw, ops.linear_prepack(pw, self.out_features, self.in_features, self.bits))
        return tiled

    def forward(self, x: torch.Tensor, residual: torch.Tensor | None = None) -> torch.Tensor:
        buffers = self._buffers
        try:       # past nn.Module's attribute protocol, 0.2 us a call
            packed, book, bias = buffers["packed_weight"], buffers["codebook"], buffers["bias"]
        except KeyError:       # one has become a parameter, or a parametrised property
            packed, book, bias = self.packed_weight, self.codebook, self.bias
        if not (self.use_cuda_kernel and x.is_cuda and packed.is_cuda):
            self._refuse()
        if self.act_scale is None:
            tiled = self._prepacked(x.numel() // self.in_features, x)
            return ops.dimq_linear_wq(x, packed, book, bias, self.out_features, self.in_features, bits=self.bits,
                                      group_rows=self.group_rows, out_dtype=self.out_dtype, epilogue=self.epilogue,
                                      residual=residual, packed_tiled=tiled)
        rows = x.numel() // self.in_features
        if rows >= ops.A4_TC_MIN_ROWS and self.in_features % 64 == 0:
            # The fp32-grade form, except for an fp32 codebook on many rows: there it multiplies two fp16 terms in
            # tiles of 128 x 128, the bf16 pair below in tiles of 256 (768 -> 3072: 20.5 against 21.1 us at 512 rows,
            # 36 / 30 at 1576; with an fp16 codebook, one term, 13.6 / 20.9 and 22 / 30, 120 / 124 for 4096 x 3072 -> 3072).
            if book.dtype != torch.float32 or rows < 1024:
                y = ops.dimq_linear_a4(x, packed, book, self.act_scale, self.act_zero_point, bias, self.out_features,
                                       self.in_features, out_dtype=self.out_dtype, epilogue=self.epilogue, residual=residual)
                if y is not None:
                    return y
            # centred activation codes (exact in bf16) times the scaled codebook through the weight-only
            # tensor-core path; per-layer state is cached, nothing is re-derived per call
            codes = ops.centre_quantize_u4(x, self.act_scale, self.act_zero_point)
            return ops.dimq_linear_wq(codes, packed, self._scaled_codebook(), bias, self.out_features, self.in_features,
                                      bits=4, out_dtype=self.out_dtype, epilogue=self.epilogue, residual=residual)
        if residual is not None or self.epilogue is not None:
            raise RuntimeError("a fused epilogue or residual needs the weight-only mode or at least "
                               f"{ops.A4_TC_MIN_ROWS} activation rows")
        return ops.dimq_linear_lut(x, packed, book, self.act_scale, self.act_zero_point, bias, self.out_features,
                                   self.in_features)

    @classmethod
    def from_export_layer(cls, layer: Mapping[str, Any], *, use_cuda_kernel: bool = True, **extra) -> "DIMQLinear":
        return cls(layer["packed_weight"], layer["codebook"], layer.get("act_scale"), layer.get("act_zero_point"),
                   layer["out_features"], layer["in_features"], layer.get("bias"), use_cuda_kernel=use_cuda_kernel,
                   bits=layer.get("bit_w", 4), group_rows=layer.get("group_rows"), **extra)

    def extra_repr(self) -> str:
        mode = "weight-only" if self.act_scale is None else "W4A4"
        return f"{self.in_features} -> {self.out_features}, bits={self.bits}, mode={mode}"


class DIMQConv2d(_PackedBase):
    """Conv2d layer backed by packed weight indices and a learned codebook."""

    def __init__(self, packed_weight, codebook, act_scale, act_zero_point, weight_shape, bias=None, *, stride=1,
                 padding=0, dilation=1, groups: int = 1, use_cuda_kernel: bool = True, bits: int = 4,
                 group_rows: int | None = None, out_dtype: torch.dtype | None = None,
                 epilogue: str | None = None) -> None:
        super().__init__()
        self._init_common(packed_weight, codebook, act_scale, act_zero_point, bias, use_cuda_kernel, bits,
                          group_rows, out_dtype, epilogue)
        self.weight_shape = tuple(int(v) for v in weight_shape)
        self.stride = _pair(stride)
        self.padding = _pair(padding)
        self.dilation = _pair(dilation)
        self.groups = int(groups)
        # indices re-ordered for the tensor-core conv: built on first use on the GPU and rebuilt
        # whenever the packed_weight buffer is replaced, moved or written in place
        self._khwc = None

    def _prepacked(self) -> torch.Tensor | None:
        if self.groups != 1 or self.weight_shape[1] % 64 != 0:
            return None
        pw = self._buffers.get("packed_weight")
        if pw is None:
            pw = self.packed_weight
        khwc = self._kept("_khwc", pw)
        if khwc is None:
            khwc = self._keep("_khwc", pw, ops.conv_prepack(pw, self.weight_shape, self.bits))
        return khwc

    def forward(self, x: torch.Tensor, residual: torch.Tensor | None = None) -> torch.Tensor:
        buffers = self._buffers
        try:       # past nn.Module's attribute protocol, 0.2 us a call
            packed, book, bias = buffers["packed_weight"], buffers["codebook"], buffers["bias"]
        except KeyError:       # one has become a parameter, or a parametrised property
            packed, book, bias = self.packed_weight, self.codebook, self.bias
        if not (self.use_cuda_kernel and x.is_cuda and packed.is_cuda):
            self._refuse()
        if self.act_scale is None:
            return ops.dimq_conv2d_wq(x, packed, book, bias, self.weight_shape, self.stride, self.padding, self.dilation,
                                      self.groups, bits=self.bits, group_rows=self.group_rows, out_dtype=self.out_dtype,
                                      epilogue=self.epilogue, residual=residual, packed_khwc=self._prepacked())
        tc = self.groups == 1 and self.weight_shape[1] % 64 == 0
        channels_last = x.dim() == 4 and x.is_contiguous(memory_format=torch.channels_last) and not x.is_contiguous()
        if tc and channels_last and self.stride[0] == self.stride[1] and self.stride[0] in (1, 2):
            oh = (x.shape[2] + 2 * self.padding[0] - self.dilation[0] * (self.weight_shape[2] - 1) - 1) // self.stride[0] + 1
            ow = (x.shape[3] + 2 * self.padding[1] - self.dilation[1] * (self.weight_shape[3] - 1) - 1) // self.stride[1] + 1
            if x.shape[0] * oh * ow >= ops.A4_TC_MIN_ROWS:
                khwc = self._prepacked()
                # fp16 / bf16 codebooks are one exact term: the fp32-grade form (64 x 64 channels on 56^2, batch 64:
                # 66 us, the bf16 pair 82; 512 on 7^2: 35 / 52); an fp32 codebook takes two there (94 / 82, 60 / 52)
                if book.dtype != torch.float32:
                    y = ops.dimq_conv2d_a4(x, packed, book, self.act_scale, self.act_zero_point, bias, self.weight_shape,
                                           self.stride, self.padding, self.dilation, self.groups, out_dtype=self.out_dtype,
                                           epilogue=self.epilogue, residual=residual, packed_khwc=khwc)
                    if y is not None:
                        return y
                # centred activation codes times the scaled codebook through the weight-only implicit-GEMM path,
                # with the re-ordered indices and the scaled codebook cached on the module
                codes = ops.centre_quantize_u4(x, self.act_scale, self.act_zero_point)
                return ops.dimq_conv2d_wq(codes, packed, self._scaled_codebook(), bias,
                                          self.weight_shape, self.stride, self.padding, self.dilation, self.groups,
                                          bits=4, out_dtype=self.out_dtype, epilogue=self.epilogue, residual=residual,
                                          packed_khwc=khwc)
        if residual is not None or self.epilogue is not None:
            raise RuntimeError("a fused epilogue or residual needs the weight-only mode, or channels_last input "
                               f"with at least {ops.A4_TC_MIN_ROWS} output pixels")
        if tc and x.dim() == 4 and _eager(x, book, bias):
            # NCHW activations, or few pixels: the re-ordered indices are kept here, not re-derived per call.  A captured
            # graph re-derives them in every replay: it follows packed_weight itself, as dimq_conv2d_lut does.
            khwc = None if _lib.host().capturing(x.get_device()) else self._prepacked()
            y = ops.dimq_conv2d_a4(x, packed, book, self.act_scale, self.act_zero_point, bias,
                                   self.weight_shape, self.stride, self.padding, self.dilation, self.groups,
                                   packed_khwc=khwc)
            if y is not None:
                return y
        return ops.dimq_conv2d_lut(x, packed, book, self.act_scale, self.act_zero_point, bias, self.weight_shape, self.stride,
                                   self.padding, self.dilation, self.groups)

    @classmethod
    def from_export_layer(cls, layer: Mapping[str, Any], *, use_cuda_kernel: bool = True, **extra) -> "DIMQConv2d":
        return cls(layer["packed_weight"], layer["codebook"], layer.get("act_scale"), layer.get("act_zero_point"),
                   layer["weight_shape"], layer.get("bias"), stride=layer.get("stride", (1, 1)),
                   padding=layer.get("padding", (0, 0)), dilation=layer.get("dilation", (1, 1)),
                   groups=layer.get("groups", 1), use_cuda_kernel=use_cuda_kernel, bits=layer.get("bit_w", 4),
                   group_rows=layer.get("group_rows"), **extra)

    def extra_repr(self) -> str:
        mode = "weight-only" if self.act_scale is None else "W4A4"
        return f"weight_shape={self.weight_shape}, stride={self.stride}, bits={self.bits}, mode={mode}"


def make_packed_layer(layer: Mapping[str, Any], *, use_cuda_kernel: bool = True, **extra) -> nn.Module:
    if layer["type"] == "linear":
        return DIMQLinear.from_export_layer(layer, use_cuda_kernel=use_cuda_kernel, **extra)
    if layer["type"] == "conv2d":
        return DIMQConv2d.from_export_layer(layer, use_cuda_kernel=use_cuda_kernel, **extra)
    raise ValueError(f"unsupported packed DIMQ layer type {layer['type']!r}")


def replace_modules_with_packed_dimq(model: nn.Module, packed_state: Mapping[str, Any], *,
                                     use_cuda_kernel: bool = True, **extra) -> nn.Module:
    """Replace matching modules in ``model`` with packed DIMQ runtime layers
    (dimq_backend/modules.py:161-172).  As in the reference, the non-quantised
    tensors of the checkpoint are not loaded here."""
    for name, layer in packed_state["layers"].items():
        parts = name.split(".")
        parent = model
        for part in parts[:-1]:
            parent = parent._modules[part]
        parent._modules[parts[-1]] = make_packed_layer(layer, use_cuda_kernel=use_cuda_kernel, **extra)
    return model
