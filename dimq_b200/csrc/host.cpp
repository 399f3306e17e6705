// Native host path of the Python entry points (dimq_b200/ops.py): argument checks, output and scratch allocation on
// PyTorch's allocator, the current stream, and the calls into libdimq_b200.so - one call from Python per operator.
//
// Why native: the kernels of a small call run 4-15 us, while the same steps in Python (ctypes argument objects, device
// context, two allocations, struct set-up) took ~30 us per call, so decoding and small-batch layers waited for the
// host: 1 x 1024 -> 4096 took 30 us per call around a 4 us kernel.  The checks, their order and their messages are
// those of the Python code they replace; every entry point keeps no state between calls.
//
// The C ABI stays the boundary: this file contains no kernel and nothing below include/dimq_b200.h knows PyTorch.
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/utils/pybind.h>

#include <ATen/ATen.h>
#include <torch/library.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>

#include <cmath>
#include <optional>
#include <stdexcept>
#include <string>

#include "../../include/dimq_b200.h"

namespace {

using at::Tensor;
using OptTensor = std::optional<Tensor>;

[[noreturn]] void fail(const std::string& msg) { throw std::runtime_error(msg); }

void require_cuda(const Tensor& t, const char* what) {
  if (!t.is_cuda()) fail(std::string(what) + " expects a CUDA tensor");
}

// The kernels get raw pointers: every operand has to be where x is.
void same_device(const Tensor& t, const Tensor& x, const char* what) {
  if (t.device() != x.device()) fail(std::string(what) + " must be on the device of the input, " + x.device().str() + ", got " + t.device().str());
}

int dtype_code(const Tensor& t, const char* what) {
  switch (t.scalar_type()) {
    case at::kFloat: return DIMQ_F32;
    case at::kHalf: return DIMQ_F16;
    case at::kBFloat16: return DIMQ_BF16;
    default: fail(std::string(what) + " must be float32, float16 or bfloat16, got " + c10::toString(t.scalar_type()));
  }
}

void check_qparams(double scale, int64_t zp) {
  if (!(scale > 0.0)) fail("act_scale must be positive");
  if (zp < 0 || zp > 15) fail("act_zero_point must be in [0, 15]");
}

// ---- Python arguments -----------------------------------------------------------------------------

const Tensor& as_tensor(PyObject* o) {
  if (!THPVariable_Check(o)) throw torch::TypeError(std::string("expected a tensor, got ") + Py_TYPE(o)->tp_name);
  return THPVariable_Unpack(o);
}

OptTensor as_opt_tensor(PyObject* o) {
  if (o == Py_None) return std::nullopt;
  return as_tensor(o);
}

int64_t as_int(PyObject* o) {
  if (PyLong_Check(o)) {
    const long long v = PyLong_AsLongLong(o);
    if (v == -1 && PyErr_Occurred()) throw python_error();
    return v;
  }
  PyObject* i = PyNumber_Long(o);     // int(o)
  if (i == nullptr) throw python_error();
  const long long v = PyLong_AsLongLong(i);
  Py_DECREF(i);
  if (v == -1 && PyErr_Occurred()) throw python_error();
  return v;
}

std::optional<int64_t> as_opt_int(PyObject* o) {
  if (o == Py_None) return std::nullopt;
  return as_int(o);
}

double as_double(PyObject* o) {
  const double v = PyFloat_AsDouble(o);
  if (v == -1.0 && PyErr_Occurred()) throw python_error();
  return v;
}

at::ScalarType as_dtype(PyObject* o) {
  if (o == Py_None) return at::kFloat;
  if (!THPDtype_Check(o)) throw torch::TypeError(std::string("expected a torch.dtype, got ") + Py_TYPE(o)->tp_name);
  return reinterpret_cast<THPDtype*>(o)->scalar_type;
}

void as_pair(PyObject* o, int32_t* a, int32_t* b) {
  if (PyLong_Check(o)) {
    *a = *b = static_cast<int32_t>(as_int(o));
    return;
  }
  PyObject* seq = PySequence_Fast(o, "expected an int or a pair");
  if (seq == nullptr) throw python_error();
  if (PySequence_Fast_GET_SIZE(seq) != 2) {
    Py_DECREF(seq);
    PyErr_Format(PyExc_ValueError, "expected pair, got %R", o);
    throw python_error();
  }
  PyObject* items[2] = {PySequence_Fast_GET_ITEM(seq, 0), PySequence_Fast_GET_ITEM(seq, 1)};
  try {
    *a = static_cast<int32_t>(as_int(items[0]));
    *b = static_cast<int32_t>(as_int(items[1]));
  } catch (...) {
    Py_DECREF(seq);
    throw;
  }
  Py_DECREF(seq);
}

void as_weight_shape(PyObject* o, int32_t (&s)[4]) {
  PyObject* seq = PySequence_Fast(o, "weight_shape must be a sequence of four sizes");
  if (seq == nullptr) throw python_error();
  if (PySequence_Fast_GET_SIZE(seq) != 4) {
    Py_DECREF(seq);
    PyErr_SetString(PyExc_ValueError, "weight_shape must have four sizes");
    throw python_error();
  }
  try {
    for (int i = 0; i < 4; ++i) s[i] = static_cast<int32_t>(as_int(PySequence_Fast_GET_ITEM(seq, i)));
  } catch (...) {
    Py_DECREF(seq);
    throw;
  }
  Py_DECREF(seq);
}

void want_args(Py_ssize_t got, Py_ssize_t want, const char* name) {
  if (got != want) throw torch::TypeError(std::string(name) + " takes " + std::to_string(want) + " arguments, got " + std::to_string(got));
}

PyObject* wrap(const OptTensor& t) {
  if (!t.has_value()) Py_RETURN_NONE;
  return THPVariable_Wrap(*t);
}

// ---- launch bookkeeping ---------------------------------------------------------------------------

PyObject* g_launch_count = nullptr;   // the list `_lib.LAUNCH_COUNT`: kernels launched by this process

void count_launches(int n) {          // GIL held
  if (g_launch_count == nullptr || n == 0) return;
  const long v = PyLong_AsLong(PyList_GET_ITEM(g_launch_count, 0));
  PyObject* nv = PyLong_FromLong(v + n);
  if (nv == nullptr || PyList_SetItem(g_launch_count, 0, nv) != 0) throw python_error();
}

PyObject* g_ops = nullptr;            // the namespace of dimq_b200.ops, which states the rules both sides follow

int64_t a4_tc_min_rows() {            // GIL not held
  pybind11::gil_scoped_acquire gil;
  PyObject* v = g_ops != nullptr ? PyDict_GetItemString(g_ops, "A4_TC_MIN_ROWS") : nullptr;
  if (v == nullptr) fail("dimq_b200.ops.A4_TC_MIN_ROWS is missing");
  return as_int(v);
}

void check(int status, const char* what) {
  if (status != DIMQ_OK)
    fail(std::string("dimq_b200.") + what + " failed: " + dimq_status_string(status) + " (status " + std::to_string(status) + ")");
}

void* stream_of(const Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }

Tensor scratch(int64_t bytes, const Tensor& like) { return at::empty({bytes}, like.options().dtype(at::kByte)); }

const void* ptr(const OptTensor& t) { return t.has_value() ? t->data_ptr() : nullptr; }

// ---- shared operand checks ------------------------------------------------------------------------

struct Weight {
  Tensor pw, cb;
  OptTensor second;      // re-ordered copy of the indices
  dimq_wq_weight w;
};

Weight wq_weight(const Tensor& x, const Tensor& packed, const Tensor& books, int64_t bits, int64_t out_rows, int64_t numel,
                 std::optional<int64_t> group_rows, const OptTensor& second) {
  require_cuda(packed, "weight-only op");
  require_cuda(books, "weight-only op");
  same_device(packed, x, "packed_weight");
  same_device(books, x, "codebook");
  if (packed.scalar_type() != at::kByte) fail("packed_weight must be uint8");
  if (!at::isFloatingType(books.scalar_type())) fail("codebook must be floating point");
  if (bits != 2 && bits != 3 && bits != 4 && bits != 8) fail("unsupported weight bit width " + std::to_string(bits));
  Weight r;
  r.pw = packed.contiguous();
  const int64_t need = (numel * bits + 7) / 8;
  if (r.pw.numel() < need) fail("packed_weight is too small for the weight shape");
  r.cb = books.contiguous();
  if (r.cb.dim() != 1 && r.cb.dim() != 2) fail("codebooks must be [entries] or [groups, entries]");
  const int64_t groups = r.cb.dim() == 1 ? 1 : r.cb.size(0), entries = r.cb.size(-1);
  if (entries > (int64_t(1) << bits)) fail(std::to_string(entries) + " codebook entries do not fit " + std::to_string(bits) + "-bit indices");
  int64_t grp = out_rows;
  if (groups != 1) {
    if (!group_rows.has_value()) fail("grouped codebooks need group_rows");
    grp = *group_rows;
    if (groups * grp < out_rows) fail("not enough codebooks for the output rows");
  }
  if (second.has_value()) {
    r.second = second->contiguous();
    if (r.second->scalar_type() != at::kByte || !r.second->is_cuda() || r.second->numel() < need)
      fail("packed_khwc must be a CUDA uint8 tensor as large as packed_weight");
    same_device(*r.second, x, "packed_khwc");
  }
  r.w.packed = static_cast<const uint8_t*>(r.pw.data_ptr());
  r.w.bits = static_cast<int32_t>(bits);
  r.w.codebooks = r.cb.data_ptr();
  r.w.cb_dtype = dtype_code(r.cb, "codebook");
  r.w.entries = static_cast<int32_t>(entries);
  r.w.groups = groups;
  r.w.group_rows = grp;
  r.w.packed_khwc = r.second.has_value() ? static_cast<const uint8_t*>(r.second->data_ptr()) : nullptr;
  return r;
}

struct Bias {
  OptTensor t;
  int dtype = 0;
};

Bias bias_arg(const OptTensor& bias, const Tensor& x, int64_t n, const char* what) {
  Bias b;
  if (!bias.has_value()) return b;
  if (!bias->is_cuda()) fail("bias must be CUDA when provided");
  same_device(*bias, x, "bias");
  if (bias->numel() != n) fail(std::string("bias numel must equal ") + what);
  b.t = bias->contiguous();
  b.dtype = dtype_code(*b.t, "bias");
  return b;
}

std::vector<int64_t> out_shape(const Tensor& x, int64_t n) {
  std::vector<int64_t> s(x.sizes().begin(), x.sizes().end());
  s.back() = n;
  return s;
}

OptTensor linear_residual(const OptTensor& residual, const Tensor& y) {
  if (!residual.has_value()) return std::nullopt;
  if (residual->scalar_type() != y.scalar_type() || residual->numel() != y.numel())
    fail("residual must match the output shape and dtype");
  same_device(*residual, y, "residual");
  return residual->contiguous();
}

// ---- linear ---------------------------------------------------------------------------------------

Tensor linear_wq(const Tensor& x, const Tensor& packed, const Tensor& books, const OptTensor& bias, int64_t n, int64_t k,
                 int64_t bits, std::optional<int64_t> group_rows, at::ScalarType out_dtype, int epilogue,
                 const OptTensor& residual, const OptTensor& tiled, int* launches) {
  require_cuda(x, "linear_wq");
  if (!at::isFloatingType(x.scalar_type())) fail("linear_wq expects floating input");
  if (n <= 0 || k <= 0) fail("linear dimensions must be positive");
  if (x.dim() == 0 || x.size(-1) != k) fail("input last dimension must equal in_features");
  const Tensor xc = x.contiguous();
  Weight w = wq_weight(x, packed, books, bits, n, n * k, group_rows, tiled);
  const Bias b = bias_arg(bias, x, n, "out_features");
  const c10::cuda::CUDAGuard guard(x.device());
  Tensor y = at::empty(out_shape(x, n), x.options().dtype(out_dtype).memory_format(at::MemoryFormat::Contiguous));
  const OptTensor res = linear_residual(residual, y);
  const int64_t m = xc.numel() / k;
  const int xd = dtype_code(xc, "x"), yd = dtype_code(y, "y");
  void* st = stream_of(x);
  // Regimes that need scratch: a few activation rows against a large weight (the k slices of the small-M kernel meet
  // there), many activation rows (the indices are expanded once to a 16-bit weight), fp32 activations (split into
  // fp16 terms) and a few hundred rows against a long K (split-K partial tiles).
  int64_t need = 0;
  int kernels = 0;
  dimq_linear_wq_ws_plan(xc.data_ptr(), xd, &w.w, ptr(res), y.data_ptr(), yd, m, n, k, -1, &need, &kernels);
  if (need > 0) {
    Tensor ws = scratch(need, x);
    check(dimq_linear_wq_ws(xc.data_ptr(), xd, &w.w, ptr(b.t), b.dtype, ptr(res), y.data_ptr(), yd, m, n, k, epilogue,
                            ws.data_ptr(), need, st), "linear_wq_ws");
    *launches = kernels;    // expansion + GEMM, GEMM + the kernel that finishes the sums, or a GEMM alone
    return y;
  }
  check(dimq_linear_wq(xc.data_ptr(), xd, &w.w, ptr(b.t), b.dtype, ptr(res), y.data_ptr(), yd, m, n, k, epilogue,
                       DIMQ_ALGO_AUTO, st), "linear_wq");
  *launches = 1;
  return y;
}

// W4A4 at fp32 grade into y; false where that form does not apply
bool linear_a4_into(const Tensor& xc, Weight& w, double scale, int64_t zp, const Bias& b, const OptTensor& res, Tensor& y,
                    int64_t m, int64_t n, int64_t k, int epilogue, int* launches) {
  const int yd = dtype_code(y, "y");
  int64_t need = 0;
  dimq_linear_a4_workspace_bytes(&w.w, yd, m, n, k, &need);
  if (need == 0) return false;
  const int xd = dtype_code(xc, "x");
  Tensor ws = scratch(need, xc);
  const int st = dimq_linear_a4(xc.data_ptr(), xd, &w.w, static_cast<float>(scale), static_cast<int>(zp), ptr(b.t), b.dtype,
                                ptr(res), y.data_ptr(), yd, m, n, k, epilogue, ws.data_ptr(), need, stream_of(xc));
  if (st == DIMQ_ERR_UNSUPPORTED) return false;
  check(st, "linear_a4");
  *launches = 2;      // the operand preparation and the GEMM
  return true;
}

OptTensor linear_a4(const Tensor& x, const Tensor& packed, const Tensor& book, double scale, int64_t zp, const OptTensor& bias,
                    int64_t n, int64_t k, at::ScalarType out_dtype, int epilogue, const OptTensor& residual, int* launches) {
  require_cuda(x, "linear_a4");
  if (!at::isFloatingType(x.scalar_type())) fail("linear_a4 expects floating input");
  check_qparams(scale, zp);
  if (n <= 0 || k <= 0) fail("linear dimensions must be positive");
  if (x.dim() == 0 || x.size(-1) != k) fail("input last dimension must equal in_features");
  Weight w = wq_weight(x, packed, book, 4, n, n * k, std::nullopt, std::nullopt);
  const Tensor xc = x.contiguous();
  const Bias b = bias_arg(bias, x, n, "out_features");
  const c10::cuda::CUDAGuard guard(x.device());
  Tensor y = at::empty(out_shape(x, n), x.options().dtype(out_dtype).memory_format(at::MemoryFormat::Contiguous));
  const OptTensor res = linear_residual(residual, y);
  if (!linear_a4_into(xc, w, scale, zp, b, res, y, xc.numel() / k, n, k, epilogue, launches)) return std::nullopt;
  return y;
}

// The reference's linear_lut: fp32 output, one 16-entry codebook.
Tensor linear_lut(const Tensor& x, const Tensor& packed, const Tensor& book, double scale, int64_t zp, const OptTensor& bias,
                  int64_t n, int64_t k, int* launches) {
  require_cuda(x, "linear_lut");
  require_cuda(packed, "linear_lut");
  require_cuda(book, "linear_lut");
  if (!at::isFloatingType(x.scalar_type())) fail("linear_lut expects floating input");
  if (packed.scalar_type() != at::kByte) fail("packed_weight must be uint8");
  if (!at::isFloatingType(book.scalar_type())) fail("codebook must be floating point");
  if (book.numel() != 16) fail("codebook must have 16 entries for W4");
  check_qparams(scale, zp);
  if (n <= 0 || k <= 0) fail("linear dimensions must be positive");
  if (x.numel() % k != 0) fail("input numel must be divisible by in_features");
  if (packed.numel() < (n * k + 1) / 2) fail("packed_weight is too small for out_features * in_features");
  if (x.dim() == 0 || x.size(-1) != k) fail("input last dimension must equal in_features");
  const Tensor xc = x.contiguous();
  Weight w = wq_weight(x, packed, book.contiguous().view(-1), 4, n, n * k, std::nullopt, std::nullopt);
  const Bias b = bias_arg(bias, x, n, "out_features");
  const c10::cuda::CUDAGuard guard(x.device());
  Tensor y = at::empty(out_shape(x, n), x.options().dtype(at::kFloat).memory_format(at::MemoryFormat::Contiguous));
  const int64_t m = xc.numel() / k;
  if (linear_a4_into(xc, w, scale, zp, b, std::nullopt, y, m, n, k, DIMQ_EPI_NONE, launches)) return y;
  const int xd = dtype_code(xc, "x");
  void* st = stream_of(x);
  if (k % 64 == 0 && reinterpret_cast<uintptr_t>(w.pw.data_ptr()) % 16 == 0 && m >= a4_tc_min_rows()) {
    int64_t need = 0;
    check(dimq_a4_workspace_bytes(xc.numel(), 0, &need), "a4_workspace_bytes");
    Tensor ws = scratch(need, x);
    const int rc = dimq_linear_lut_tc(xc.data_ptr(), xd, w.w.packed, w.w.codebooks, w.w.cb_dtype, static_cast<float>(scale),
                                      static_cast<int>(zp), ptr(b.t), b.dtype, static_cast<float*>(y.data_ptr()), m, n, k,
                                      ws.data_ptr(), need, st);
    if (rc != DIMQ_ERR_UNSUPPORTED) {
      check(rc, "linear_lut_tc");
      *launches = 2;  // the activation quantiser and the GEMM
      return y;
    }
  }
  check(dimq_linear_lut(xc.data_ptr(), xd, w.w.packed, w.w.codebooks, w.w.cb_dtype, static_cast<float>(scale),
                        static_cast<int>(zp), ptr(b.t), b.dtype, static_cast<float*>(y.data_ptr()), m, n, k, st), "linear_lut");
  *launches = 1;
  return y;
}

// ---- convolution ----------------------------------------------------------------------------------

struct ConvArgs {
  int32_t shape[4];
  int32_t sh, sw, ph, pw, dh, dw;
  int64_t groups;
};

dimq_conv_geom conv_geom(const Tensor& x, const ConvArgs& a) {
  dimq_conv_geom g;
  memset(&g, 0, sizeof(g));
  g.batch = static_cast<int32_t>(x.size(0));
  g.in_channels = static_cast<int32_t>(x.size(1));
  g.in_h = static_cast<int32_t>(x.size(2));
  g.in_w = static_cast<int32_t>(x.size(3));
  g.out_channels = a.shape[0];
  g.in_channels_per_group = a.shape[1];
  g.kernel_h = a.shape[2];
  g.kernel_w = a.shape[3];
  g.stride_h = a.sh; g.stride_w = a.sw;
  g.pad_h = a.ph; g.pad_w = a.pw;
  g.dilation_h = a.dh; g.dilation_w = a.dw;
  g.groups = static_cast<int32_t>(a.groups);
  if (g.out_channels <= 0 || g.in_channels_per_group <= 0) fail("channel counts must be positive");
  if (g.kernel_h <= 0 || g.kernel_w <= 0) fail("kernel size must be positive");
  if (g.stride_h <= 0 || g.stride_w <= 0) fail("stride must be positive");
  if (g.dilation_h <= 0 || g.dilation_w <= 0) fail("dilation must be positive");
  if (g.groups <= 0) fail("groups must be positive");
  if (g.in_channels != g.in_channels_per_group * g.groups) fail("input channels do not match weight/groups");
  if (g.out_channels % g.groups != 0) fail("out_channels must be divisible by groups");
  if (dimq_conv_out_size(&g) != DIMQ_OK) fail("computed negative output size");
  return g;
}

// Input as stored (NCHW-contiguous or channels_last, no copy) and an output in the same format.
Tensor conv_io(const Tensor& x, dimq_conv_geom& g, at::ScalarType out_dtype, Tensor& y) {
  const bool contiguous = x.is_contiguous();
  const bool channels_last = !contiguous && x.is_contiguous(at::MemoryFormat::ChannelsLast);
  const Tensor xc = channels_last || contiguous ? x : x.contiguous();
  y = at::empty({g.batch, g.out_channels, g.out_h, g.out_w},
                x.options().dtype(out_dtype).memory_format(channels_last ? at::MemoryFormat::ChannelsLast : at::MemoryFormat::Contiguous));
  for (int i = 0; i < 4; ++i) {
    g.x_stride[i] = xc.stride(i);
    g.y_stride[i] = y.stride(i);
  }
  return xc;
}

void conv_residual(const OptTensor& residual, const Tensor& y) {
  if (residual.has_value() && (residual->scalar_type() != y.scalar_type() || residual->sizes() != y.sizes() ||
                               residual->strides() != y.strides()))
    fail("residual must match the output shape, dtype and memory format");
  if (residual.has_value()) same_device(*residual, y, "residual");
}

int64_t weight_numel(const dimq_conv_geom& g) {
  return static_cast<int64_t>(g.out_channels) * g.in_channels_per_group * g.kernel_h * g.kernel_w;
}

Tensor conv2d_wq(const Tensor& x, const Tensor& packed, const Tensor& books, const OptTensor& bias, const ConvArgs& a,
                 int64_t bits, std::optional<int64_t> group_rows, at::ScalarType out_dtype, int epilogue,
                 const OptTensor& residual, const OptTensor& khwc, int* launches) {
  require_cuda(x, "conv2d_wq");
  if (x.dim() != 4) fail("conv2d_wq expects NCHW input");
  if (!at::isFloatingType(x.scalar_type())) fail("conv2d_wq expects floating input");
  dimq_conv_geom g = conv_geom(x, a);
  Weight w = wq_weight(x, packed, books, bits, g.out_channels, weight_numel(g), group_rows, khwc);
  const Bias b = bias_arg(bias, x, g.out_channels, "out_channels");
  const c10::cuda::CUDAGuard guard(x.device());
  Tensor y;
  const Tensor xc = conv_io(x, g, out_dtype, y);
  if (y.numel() == 0) return y;
  conv_residual(residual, y);
  const int xd = dtype_code(xc, "x"), yd = dtype_code(y, "y");
  void* st = stream_of(x);
  // Many output pixels: the indices are expanded once to a 16-bit weight in scratch for a dense tensor-core kernel -
  // the implicit GEMM over the re-ordered indices, or the stem kernel for a 3-channel stride-2 convolution.
  // They write the activations' type or fp32.
  int64_t need = 0;
  if (yd == xd || yd == DIMQ_F32) dimq_conv2d_wq_workspace_bytes(xc.data_ptr(), xd, &w.w, &g, &need);
  if (need > 0) {
    Tensor ws = scratch(need, x);
    check(dimq_conv2d_wq_ws(xc.data_ptr(), xd, &w.w, ptr(b.t), b.dtype, ptr(residual), y.data_ptr(), yd, &g, epilogue,
                            ws.data_ptr(), need, st), "conv2d_wq_ws");
    *launches = 2;    // the expansion and the convolution
    return y;
  }
  check(dimq_conv2d_wq(xc.data_ptr(), xd, &w.w, ptr(b.t), b.dtype, ptr(residual), y.data_ptr(), yd, &g, epilogue,
                       DIMQ_ALGO_AUTO, st), "conv2d_wq");
  *launches = 1;
  return y;
}

// W4A4 at fp32 grade into y; false where that form does not apply.  w.second: the re-ordered indices, if kept.
bool conv2d_a4_into(const Tensor& xc, Weight& w, double scale, int64_t zp, const Bias& b, const OptTensor& res, Tensor& y,
                    const dimq_conv_geom& g, int epilogue, int* launches) {
  if (g.groups != 1 || g.in_channels % 64 != 0) return false;
  const int yd = dtype_code(y, "y");
  const bool kept = w.second.has_value();
  if (!kept) w.w.packed_khwc = w.w.packed;          // a stand-in for the size query
  int64_t need = 0;
  dimq_conv2d_a4_workspace_bytes(&w.w, yd, &g, &need);
  if (!kept) w.w.packed_khwc = nullptr;
  if (need == 0) return false;
  const int xd = dtype_code(xc, "x");
  void* st = stream_of(xc);
  if (!kept) {
    w.second = scratch((weight_numel(g) * 4 + 7) / 8, xc);
    uint8_t* dst = static_cast<uint8_t*>(w.second->data_ptr());
    check(dimq_conv_prepack(w.w.packed, 4, g.out_channels, g.in_channels_per_group, g.kernel_h, g.kernel_w, dst, st), "conv_prepack");
    *launches += 1;
    w.w.packed_khwc = dst;
  }
  Tensor ws = scratch(need, xc);
  const int rc = dimq_conv2d_a4(xc.data_ptr(), xd, &w.w, static_cast<float>(scale), static_cast<int>(zp), ptr(b.t), b.dtype,
                                ptr(res), y.data_ptr(), yd, &g, epilogue, ws.data_ptr(), need, st);
  if (rc == DIMQ_ERR_UNSUPPORTED) return false;
  check(rc, "conv2d_a4");
  *launches += 2;     // the operand preparation and the convolution
  return true;
}

OptTensor conv2d_a4(const Tensor& x, const Tensor& packed, const Tensor& book, double scale, int64_t zp, const OptTensor& bias,
                    const ConvArgs& a, at::ScalarType out_dtype, int epilogue, const OptTensor& residual,
                    const OptTensor& khwc, int* launches) {
  require_cuda(x, "conv2d_a4");
  if (x.dim() != 4) fail("conv2d_a4 expects NCHW input");
  if (!at::isFloatingType(x.scalar_type())) fail("conv2d_a4 expects floating input");
  check_qparams(scale, zp);
  dimq_conv_geom g = conv_geom(x, a);
  Weight w = wq_weight(x, packed, book, 4, g.out_channels, weight_numel(g), std::nullopt, khwc);
  const Bias b = bias_arg(bias, x, g.out_channels, "out_channels");
  const c10::cuda::CUDAGuard guard(x.device());
  Tensor y;
  const Tensor xc = conv_io(x, g, out_dtype, y);
  if (y.numel() == 0) return y;
  conv_residual(residual, y);
  if (!conv2d_a4_into(xc, w, scale, zp, b, residual, y, g, epilogue, launches)) return std::nullopt;
  return y;
}

// The reference's conv2d_lut: fp32 output, one 16-entry codebook.
Tensor conv2d_lut(const Tensor& x, const Tensor& packed, const Tensor& book, double scale, int64_t zp, const OptTensor& bias,
                  const ConvArgs& a, int* launches) {
  require_cuda(x, "conv2d_lut");
  if (x.dim() != 4) fail("conv2d_lut expects NCHW input");
  require_cuda(packed, "conv2d_lut");
  require_cuda(book, "conv2d_lut");
  if (!at::isFloatingType(x.scalar_type())) fail("conv2d_lut expects floating input");
  if (packed.scalar_type() != at::kByte) fail("packed_weight must be uint8");
  if (!at::isFloatingType(book.scalar_type())) fail("codebook must be floating point");
  if (book.numel() != 16) fail("codebook must have 16 entries for W4");
  check_qparams(scale, zp);
  dimq_conv_geom g = conv_geom(x, a);
  const int64_t numel = weight_numel(g);
  if (packed.numel() < (numel + 1) / 2) fail("packed_weight is too small for requested conv weight shape");
  const Bias b = bias_arg(bias, x, g.out_channels, "out_channels");
  const c10::cuda::CUDAGuard guard(x.device());
  Tensor y;
  const Tensor xc = conv_io(x, g, at::kFloat, y);
  if (y.numel() == 0) return y;
  Weight w = wq_weight(x, packed, book.contiguous().view(-1), 4, g.out_channels, numel, std::nullopt, std::nullopt);
  if (conv2d_a4_into(xc, w, scale, zp, b, std::nullopt, y, g, DIMQ_EPI_NONE, launches)) return y;
  const int xd = dtype_code(xc, "x");
  void* st = stream_of(x);
  float* yp = static_cast<float*>(y.data_ptr());
  if (g.x_stride[1] == 1 && g.y_stride[1] == 1 && g.groups == 1 && g.in_channels % 64 == 0 &&
      static_cast<int64_t>(g.batch) * g.out_h * g.out_w >= a4_tc_min_rows()) {
    int64_t need = 0;
    check(dimq_a4_workspace_bytes(xc.numel(), numel, &need), "a4_workspace_bytes");
    Tensor ws = scratch(need, x);
    const int rc = dimq_conv2d_lut_tc(xc.data_ptr(), xd, w.w.packed, w.w.codebooks, w.w.cb_dtype, static_cast<float>(scale),
                                      static_cast<int>(zp), ptr(b.t), b.dtype, yp, &g, ws.data_ptr(), need, st);
    if (rc != DIMQ_ERR_UNSUPPORTED) {
      check(rc, "conv2d_lut_tc");
      *launches += 3; // index re-order, activation quantiser, convolution
      return y;
    }
  }
  check(dimq_conv2d_lut(xc.data_ptr(), xd, w.w.packed, w.w.codebooks, w.w.cb_dtype, static_cast<float>(scale),
                        static_cast<int>(zp), ptr(b.t), b.dtype, yp, &g, st), "conv2d_lut");
  *launches += 1;
  return y;
}

// ---- export and quantisation-aware training -------------------------------------------------------

struct Books {
  Tensor cb;
  int64_t rows, cols, grp;
  int entries;
};

Books codebook_rows(const Tensor& wc, const Tensor& codebooks, std::optional<int64_t> group_rows, const char* what) {
  Books r;
  r.cb = codebooks.detach().to(wc.options().dtype(at::kFloat).memory_format(std::nullopt)).contiguous();
  if (r.cb.dim() == 1) r.cb = r.cb.view({1, -1});
  if (r.cb.dim() < 2) fail("codebooks must be [entries] or [groups, entries]");
  const int64_t entries = r.cb.size(1);
  if (entries == 0) fail("centers must be non-empty");
  if (entries > 256) fail(std::string(what) + " supports at most 256 centres");
  r.entries = static_cast<int>(entries);
  if (r.cb.size(0) == 1) {
    r.rows = 1;
    r.cols = wc.numel();
    r.grp = 1;
  } else {
    if (!group_rows.has_value() || wc.dim() < 1) fail("grouped codebooks need group_rows");
    r.rows = wc.size(0);
    r.cols = wc.numel() / (r.rows > 1 ? r.rows : 1);
    r.grp = *group_rows;
    if (r.cb.size(0) * r.grp < r.rows) fail("not enough codebooks for the rows of w");
  }
  return r;
}

std::pair<OptTensor, OptTensor> hard_quantize(const Tensor& w, const Tensor& codebooks, std::optional<int64_t> group_rows,
                                              std::optional<int64_t> bits, bool want_idx, int* launches) {
  require_cuda(w, "hard_quantize");
  if (!at::isFloatingType(w.scalar_type())) fail("hard_quantize expects floating weights");
  const c10::cuda::CUDAGuard guard(w.device());
  const Tensor wc = w.detach().contiguous();
  const Books q = codebook_rows(wc, codebooks, group_rows, "hard_quantize");
  if (bits.has_value()) {
    const int64_t b = *bits;
    if (!(b == 1 || b == 2 || b == 3 || b == 4 || b == 8) || q.entries > (1 << b))
      fail("cannot pack " + std::to_string(q.entries) + "-entry indices into " + std::to_string(b) + " bits");
  }
  const auto bytes = wc.options().dtype(at::kByte);
  OptTensor idx, packed;
  if (want_idx) idx = at::empty(wc.sizes(), bytes.memory_format(at::MemoryFormat::Contiguous));
  if (bits.has_value()) packed = at::empty({(wc.numel() * *bits + 7) / 8}, bytes);
  if (!idx.has_value() && !packed.has_value()) fail("nothing to compute: ask for indices, packed bytes or both");
  check(dimq_hard_quantize(wc.data_ptr(), dtype_code(wc, "w"), q.rows, q.cols, static_cast<const float*>(q.cb.data_ptr()), q.entries,
                           q.grp, idx.has_value() ? static_cast<uint8_t*>(idx->data_ptr()) : nullptr,
                           packed.has_value() ? static_cast<uint8_t*>(packed->data_ptr()) : nullptr,
                           static_cast<int>(bits.value_or(8)), stream_of(w)), "hard_quantize");
  *launches = 1;
  return {idx, packed};
}

std::pair<Tensor, OptTensor> fake_quantize_ste(const Tensor& w, const Tensor& codebooks, std::optional<int64_t> group_rows,
                                               bool want_idx, int* launches) {
  require_cuda(w, "fake_quantize_ste");
  if (!at::isFloatingType(w.scalar_type()) || w.scalar_type() == at::kDouble)
    fail("fake_quantize_ste expects float32, float16 or bfloat16 weights");
  const c10::cuda::CUDAGuard guard(w.device());
  const Tensor wc = w.detach().contiguous();
  const Books q = codebook_rows(wc, codebooks, group_rows, "fake_quantize_ste");
  Tensor out = at::empty_like(wc);
  OptTensor idx;
  if (want_idx) idx = at::empty(wc.sizes(), wc.options().dtype(at::kByte).memory_format(at::MemoryFormat::Contiguous));
  check(dimq_fake_quantize_ste(wc.data_ptr(), dtype_code(wc, "w"), q.rows, q.cols, static_cast<const float*>(q.cb.data_ptr()), q.entries,
                               q.grp, out.data_ptr(), idx.has_value() ? static_cast<uint8_t*>(idx->data_ptr()) : nullptr,
                               stream_of(w)), "fake_quantize_ste");
  *launches = 1;
  return {out, idx};
}

Tensor unpack_bits(const Tensor& packed, int64_t numel, int64_t bits, int* launches) {
  require_cuda(packed, "unpack");
  if (packed.scalar_type() != at::kByte) fail("unpack expects uint8 packed data");
  if (numel < 0) fail("numel must be non-negative");
  if (packed.numel() < (numel * bits + 7) / 8) fail("packed tensor is too small for requested numel");
  const c10::cuda::CUDAGuard guard(packed.device());
  const Tensor flat = packed.contiguous();
  Tensor out = at::empty({numel}, flat.options().memory_format(at::MemoryFormat::Contiguous));
  check(dimq_unpack_bits(static_cast<const uint8_t*>(flat.data_ptr()), numel, static_cast<int>(bits),
                         static_cast<uint8_t*>(out.data_ptr()), stream_of(packed)), "unpack_bits");
  *launches = 1;
  return out;
}

Tensor pack_bits(const Tensor& indices, int64_t bits, int* launches) {
  require_cuda(indices, "pack");
  if (indices.scalar_type() != at::kByte) fail("pack expects uint8 indices");
  const c10::cuda::CUDAGuard guard(indices.device());
  const Tensor flat = indices.contiguous();
  const int64_t n = flat.numel();
  Tensor out = at::empty({(n * bits + 7) / 8}, flat.options().memory_format(at::MemoryFormat::Contiguous));
  check(dimq_pack_bits(static_cast<const uint8_t*>(flat.data_ptr()), n, static_cast<int>(bits),
                       static_cast<uint8_t*>(out.data_ptr()), stream_of(indices)), "pack_bits");
  *launches = 1;
  return out;
}

// ---- dense helpers of the models ------------------------------------------------------------------

std::pair<Tensor, Tensor> add_layer_norm(const Tensor& x, const OptTensor& delta, const Tensor& weight, const Tensor& bias,
                                         double eps, int* launches) {
  require_cuda(x, "add_layer_norm");
  const int64_t cols = x.size(-1);
  const c10::cuda::CUDAGuard guard(x.device());
  const Tensor xc = x.contiguous();
  OptTensor dc;
  if (delta.has_value()) {
    dc = delta->contiguous();
    same_device(*dc, x, "delta");
    if (dc->sizes() != xc.sizes() || dc->scalar_type() != xc.scalar_type()) fail("delta must match x in shape and dtype");
  }
  same_device(weight, x, "weight");
  same_device(bias, x, "bias");
  const Tensor w = weight.to(xc.scalar_type()).contiguous(), b = bias.to(xc.scalar_type()).contiguous();
  if (w.numel() != cols || b.numel() != cols) fail("weight / bias must have one element per column");
  Tensor x_out = dc.has_value() ? at::empty_like(xc) : xc;
  Tensor h = at::empty_like(xc);
  check(dimq_add_layer_norm(xc.data_ptr(), ptr(dc), w.data_ptr(), b.data_ptr(), dc.has_value() ? x_out.data_ptr() : nullptr,
                            h.data_ptr(), cols == 0 ? 0 : xc.numel() / cols, cols, static_cast<float>(eps), dtype_code(xc, "x"),
                            stream_of(x)), "add_layer_norm");
  *launches = 1;
  return {x_out, h};
}

Tensor max_pool_nhwc(const Tensor& x, int64_t kernel, int64_t stride, int64_t padding, int* launches) {
  require_cuda(x, "max_pool_nhwc");
  if (x.dim() != 4 || !x.is_contiguous(at::MemoryFormat::ChannelsLast)) fail("max_pool_nhwc expects a channels_last 4-D tensor");
  if (stride == 0) fail("stride must be positive");
  const auto out = [&](int64_t v) {      // floor division, as Python's
    const int64_t q = v + 2 * padding - kernel;
    return (q >= 0 ? q / stride : -((-q + stride - 1) / stride)) + 1;
  };
  const int64_t b = x.size(0), c = x.size(1), h = x.size(2), w = x.size(3);
  const c10::cuda::CUDAGuard guard(x.device());
  Tensor y = at::empty({b, c, out(h), out(w)}, x.options().memory_format(at::MemoryFormat::ChannelsLast));
  check(dimq_max_pool_nhwc(x.data_ptr(), y.data_ptr(), dtype_code(x, "x"), b, h, w, c, static_cast<int>(kernel),
                           static_cast<int>(stride), static_cast<int>(padding), stream_of(x)), "max_pool_nhwc");
  *launches = 1;
  return y;
}

Tensor images_to_nhwc(const Tensor& x, at::ScalarType dtype, int* launches) {
  require_cuda(x, "images_to_nhwc");
  if (x.dim() != 4 || x.size(1) != 3 || !x.is_contiguous() || (x.size(2) * x.size(3)) % 8 != 0)
    fail("images_to_nhwc expects a contiguous [B, 3, H, W] tensor with H * W a multiple of 8");
  if (dtype != at::kBFloat16 && dtype != at::kHalf) fail("images_to_nhwc writes bf16 or fp16");
  const c10::cuda::CUDAGuard guard(x.device());
  Tensor y = at::empty(x.sizes(), x.options().dtype(dtype).memory_format(at::MemoryFormat::ChannelsLast));
  check(dimq_images_to_nhwc(x.data_ptr(), dtype_code(x, "images"), y.data_ptr(), dtype_code(y, "y"), x.size(0), x.size(2),
                            x.size(3), stream_of(x)), "images_to_nhwc");
  *launches = 1;
  return y;
}

Tensor attention_qkv(const Tensor& qkv, int64_t heads, int* launches) {
  require_cuda(qkv, "attention_qkv");
  if (qkv.dim() != 3 || heads <= 0 || qkv.size(2) % (3 * heads) != 0) fail("attention_qkv expects [batch, tokens, 3 * heads * head_dim]");
  const c10::cuda::CUDAGuard guard(qkv.device());
  const Tensor xc = qkv.contiguous();
  const int64_t d = xc.size(2) / (3 * heads);
  Tensor y = at::empty({xc.size(0), xc.size(1), heads * d}, xc.options().memory_format(at::MemoryFormat::Contiguous));
  check(dimq_attention_qkv(xc.data_ptr(), y.data_ptr(), xc.size(0), xc.size(1), heads, d,
                           1.0f / std::sqrt(static_cast<float>(d)), dtype_code(xc, "qkv"), stream_of(qkv)), "attention_qkv");
  *launches = 1;
  return y;
}

// ---- the Python module ----------------------------------------------------------------------------

#define ARGS(want, name) want_args(n, want, name)
#define NO_GIL pybind11::gil_scoped_release no_gil

ConvArgs conv_args(PyObject* const* a) {   // weight_shape, stride, padding, dilation, groups
  ConvArgs c;
  as_weight_shape(a[0], c.shape);
  as_pair(a[1], &c.sh, &c.sw);
  as_pair(a[2], &c.ph, &c.pw);
  as_pair(a[3], &c.dh, &c.dw);
  c.groups = as_int(a[4]);
  return c;
}

PyObject* pair_of(const OptTensor& a, const OptTensor& b) {
  PyObject* pa = wrap(a);
  PyObject* pb = wrap(b);
  PyObject* t = pa != nullptr && pb != nullptr ? PyTuple_Pack(2, pa, pb) : nullptr;
  Py_XDECREF(pa);
  Py_XDECREF(pb);
  return t;
}

PyObject* py_linear_wq(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  ARGS(12, "linear_wq");
  const Tensor x = as_tensor(a[0]), pw = as_tensor(a[1]), cb = as_tensor(a[2]);
  const OptTensor bias = as_opt_tensor(a[3]), res = as_opt_tensor(a[10]), tiled = as_opt_tensor(a[11]);
  const int64_t nf = as_int(a[4]), kf = as_int(a[5]), bits = as_int(a[6]);
  const auto grp = as_opt_int(a[7]);
  const at::ScalarType dt = as_dtype(a[8]);
  const int epi = static_cast<int>(as_int(a[9]));
  int launches = 0;
  Tensor y;
  { NO_GIL; y = linear_wq(x, pw, cb, bias, nf, kf, bits, grp, dt, epi, res, tiled, &launches); }
  count_launches(launches);
  return THPVariable_Wrap(y);
  END_HANDLE_TH_ERRORS
}

PyObject* py_linear_a4(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  ARGS(11, "linear_a4");
  const Tensor x = as_tensor(a[0]), pw = as_tensor(a[1]), cb = as_tensor(a[2]);
  const double scale = as_double(a[3]);
  const int64_t zp = as_int(a[4]), nf = as_int(a[6]), kf = as_int(a[7]);
  const OptTensor bias = as_opt_tensor(a[5]), res = as_opt_tensor(a[10]);
  const at::ScalarType dt = as_dtype(a[8]);
  const int epi = static_cast<int>(as_int(a[9]));
  int launches = 0;
  OptTensor y;
  { NO_GIL; y = linear_a4(x, pw, cb, scale, zp, bias, nf, kf, dt, epi, res, &launches); }
  count_launches(launches);
  return wrap(y);
  END_HANDLE_TH_ERRORS
}

PyObject* py_conv2d_wq(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  ARGS(15, "conv2d_wq");
  const Tensor x = as_tensor(a[0]), pw = as_tensor(a[1]), cb = as_tensor(a[2]);
  const OptTensor bias = as_opt_tensor(a[3]), res = as_opt_tensor(a[13]), khwc = as_opt_tensor(a[14]);
  const ConvArgs c = conv_args(a + 4);
  const int64_t bits = as_int(a[9]);
  const auto grp = as_opt_int(a[10]);
  const at::ScalarType dt = as_dtype(a[11]);
  const int epi = static_cast<int>(as_int(a[12]));
  int launches = 0;
  Tensor y;
  { NO_GIL; y = conv2d_wq(x, pw, cb, bias, c, bits, grp, dt, epi, res, khwc, &launches); }
  count_launches(launches);
  return THPVariable_Wrap(y);
  END_HANDLE_TH_ERRORS
}

PyObject* py_conv2d_a4(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  ARGS(15, "conv2d_a4");
  const Tensor x = as_tensor(a[0]), pw = as_tensor(a[1]), cb = as_tensor(a[2]);
  const double scale = as_double(a[3]);
  const int64_t zp = as_int(a[4]);
  const OptTensor bias = as_opt_tensor(a[5]), res = as_opt_tensor(a[13]), khwc = as_opt_tensor(a[14]);
  const ConvArgs c = conv_args(a + 6);
  const at::ScalarType dt = as_dtype(a[11]);
  const int epi = static_cast<int>(as_int(a[12]));
  int launches = 0;
  OptTensor y;
  { NO_GIL; y = conv2d_a4(x, pw, cb, scale, zp, bias, c, dt, epi, res, khwc, &launches); }
  count_launches(launches);
  return wrap(y);
  END_HANDLE_TH_ERRORS
}

PyObject* py_hard_quantize(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  ARGS(5, "hard_quantize");
  const Tensor w = as_tensor(a[0]), cb = as_tensor(a[1]);
  const auto grp = as_opt_int(a[2]), bits = as_opt_int(a[3]);
  const bool want_idx = PyObject_IsTrue(a[4]) == 1;
  int launches = 0;
  std::pair<OptTensor, OptTensor> r;
  { NO_GIL; r = hard_quantize(w, cb, grp, bits, want_idx, &launches); }
  count_launches(launches);
  return pair_of(r.first, r.second);
  END_HANDLE_TH_ERRORS
}

PyObject* py_fake_quantize_ste(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  ARGS(4, "fake_quantize_ste");
  const Tensor w = as_tensor(a[0]), cb = as_tensor(a[1]);
  const auto grp = as_opt_int(a[2]);
  const bool want_idx = PyObject_IsTrue(a[3]) == 1;
  int launches = 0;
  std::pair<Tensor, OptTensor> r;
  { NO_GIL; r = fake_quantize_ste(w, cb, grp, want_idx, &launches); }
  count_launches(launches);
  if (!want_idx) return THPVariable_Wrap(r.first);
  return pair_of(r.first, r.second);
  END_HANDLE_TH_ERRORS
}

PyObject* py_unpack_bits(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  ARGS(3, "unpack_bits");
  const Tensor packed = as_tensor(a[0]);
  const int64_t numel = as_int(a[1]), bits = as_int(a[2]);
  int launches = 0;
  Tensor y;
  { NO_GIL; y = unpack_bits(packed, numel, bits, &launches); }
  count_launches(launches);
  return THPVariable_Wrap(y);
  END_HANDLE_TH_ERRORS
}

PyObject* py_pack_bits(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  ARGS(2, "pack_bits");
  const Tensor idx = as_tensor(a[0]);
  const int64_t bits = as_int(a[1]);
  int launches = 0;
  Tensor y;
  { NO_GIL; y = pack_bits(idx, bits, &launches); }
  count_launches(launches);
  return THPVariable_Wrap(y);
  END_HANDLE_TH_ERRORS
}

PyObject* py_add_layer_norm(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  ARGS(5, "add_layer_norm");
  const Tensor x = as_tensor(a[0]), w = as_tensor(a[2]), b = as_tensor(a[3]);
  const OptTensor delta = as_opt_tensor(a[1]);
  const double eps = as_double(a[4]);
  int launches = 0;
  std::pair<Tensor, Tensor> r;
  { NO_GIL; r = add_layer_norm(x, delta, w, b, eps, &launches); }
  count_launches(launches);
  // without a delta the sum is x itself: the caller gets its own object back
  PyObject* px = !delta.has_value() && r.first.unsafeGetTensorImpl() == x.unsafeGetTensorImpl() ? Py_NewRef(a[0]) : THPVariable_Wrap(r.first);
  PyObject* ph = THPVariable_Wrap(r.second);
  PyObject* t = px != nullptr && ph != nullptr ? PyTuple_Pack(2, px, ph) : nullptr;
  Py_XDECREF(px);
  Py_XDECREF(ph);
  return t;
  END_HANDLE_TH_ERRORS
}

PyObject* py_max_pool_nhwc(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  ARGS(4, "max_pool_nhwc");
  const Tensor x = as_tensor(a[0]);
  const int64_t k = as_int(a[1]), s = as_int(a[2]), p = as_int(a[3]);
  int launches = 0;
  Tensor y;
  { NO_GIL; y = max_pool_nhwc(x, k, s, p, &launches); }
  count_launches(launches);
  return THPVariable_Wrap(y);
  END_HANDLE_TH_ERRORS
}

PyObject* py_attention_qkv(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  ARGS(2, "attention_qkv");
  const Tensor x = as_tensor(a[0]);
  const int64_t heads = as_int(a[1]);
  int launches = 0;
  Tensor y;
  { NO_GIL; y = attention_qkv(x, heads, &launches); }
  count_launches(launches);
  return THPVariable_Wrap(y);
  END_HANDLE_TH_ERRORS
}

PyObject* py_images_to_nhwc(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  ARGS(2, "images_to_nhwc");
  const Tensor x = as_tensor(a[0]);
  const at::ScalarType dt = as_dtype(a[1]);
  int launches = 0;
  Tensor y;
  { NO_GIL; y = images_to_nhwc(x, dt, &launches); }
  count_launches(launches);
  return THPVariable_Wrap(y);
  END_HANDLE_TH_ERRORS
}

// ---- torch.ops.dimq: the kernels of the CUDA key for the schemas dimq_b200/ops.py defines ---------------
// (the dispatcher calls these without the GIL)

void count_launches_no_gil(int n) {
  pybind11::gil_scoped_acquire gil;
  count_launches(n);
}

Tensor op_pack_u4(const Tensor& indices) {
  int launches = 0;
  Tensor y = pack_bits(indices, 4, &launches);
  count_launches_no_gil(launches);
  return y;
}

Tensor op_unpack_u4(const Tensor& packed, int64_t numel) {
  int launches = 0;
  Tensor y = unpack_bits(packed, numel, 4, &launches);
  count_launches_no_gil(launches);
  return y;
}

Tensor op_linear_lut(const Tensor& x, const Tensor& packed_w, const Tensor& codebook, double act_scale, int64_t act_zp,
                     const OptTensor& bias, int64_t out_features, int64_t in_features) {
  int launches = 0;
  Tensor y = linear_lut(x, packed_w, codebook, act_scale, act_zp, bias, out_features, in_features, &launches);
  count_launches_no_gil(launches);
  return y;
}

Tensor op_conv2d_lut(const Tensor& x, const Tensor& packed_w, const Tensor& codebook, double act_scale, int64_t act_zp,
                     const OptTensor& bias, int64_t out_channels, int64_t in_channels_per_group, int64_t kernel_h,
                     int64_t kernel_w, int64_t stride_h, int64_t stride_w, int64_t pad_h, int64_t pad_w, int64_t dilation_h,
                     int64_t dilation_w, int64_t groups) {
  const auto i32 = [](int64_t v) { return static_cast<int32_t>(v); };
  const ConvArgs a = {{i32(out_channels), i32(in_channels_per_group), i32(kernel_h), i32(kernel_w)}, i32(stride_h), i32(stride_w),
                      i32(pad_h), i32(pad_w), i32(dilation_h), i32(dilation_w), groups};
  int launches = 0;
  Tensor y = conv2d_lut(x, packed_w, codebook, act_scale, act_zp, bias, a, &launches);
  count_launches_no_gil(launches);
  return y;
}

TORCH_LIBRARY_IMPL(dimq, CUDA, m) {
  m.impl("pack_u4", op_pack_u4);
  m.impl("unpack_u4", op_unpack_u4);
  m.impl("linear_lut", op_linear_lut);
  m.impl("conv2d_lut", op_conv2d_lut);
}

PyObject* py_set_launch_count(PyObject*, PyObject* list) {
  if (!PyList_Check(list) || PyList_GET_SIZE(list) < 1) {
    PyErr_SetString(PyExc_TypeError, "expected a list of one integer");
    return nullptr;
  }
  Py_INCREF(list);
  Py_XSETREF(g_launch_count, list);
  Py_RETURN_NONE;
}

PyObject* py_set_ops(PyObject*, PyObject* dict) {
  if (!PyDict_Check(dict)) {
    PyErr_SetString(PyExc_TypeError, "expected the namespace of dimq_b200.ops");
    return nullptr;
  }
  Py_INCREF(dict);
  Py_XSETREF(g_ops, dict);
  Py_RETURN_NONE;
}

// ---- events of the tensors that modules keep (dimq_b200/modules.py) --------------------------------

constexpr char kEvent[] = "dimq_b200.event";

void cuda_ok(cudaError_t e, const char* what) {
  if (e != cudaSuccess) fail(std::string(what) + " failed: " + cudaGetErrorString(e));
}

cudaEvent_t as_event(PyObject* o) {
  void* e = PyCapsule_GetPointer(o, kEvent);
  if (e == nullptr) throw python_error();
  return static_cast<cudaEvent_t>(e);
}

c10::DeviceIndex as_device(PyObject* o) { return static_cast<c10::DeviceIndex>(as_int(o)); }

// a new event, recorded on the device's current stream
PyObject* py_record_event(PyObject*, PyObject* device) {
  HANDLE_TH_ERRORS
  const c10::cuda::CUDAGuard guard(as_device(device));
  cudaEvent_t e = nullptr;
  cuda_ok(cudaEventCreateWithFlags(&e, cudaEventDisableTiming), "cudaEventCreateWithFlags");
  PyObject* capsule = PyCapsule_New(e, kEvent, [](PyObject* o) {
    (void)cudaEventDestroy(static_cast<cudaEvent_t>(PyCapsule_GetPointer(o, kEvent)));
  });
  if (capsule == nullptr) {
    (void)cudaEventDestroy(e);
    throw python_error();
  }
  const cudaError_t rc = cudaEventRecord(e, c10::cuda::getCurrentCUDAStream(as_device(device)).stream());
  if (rc != cudaSuccess) Py_DECREF(capsule);
  cuda_ok(rc, "cudaEventRecord");
  return capsule;
  END_HANDLE_TH_ERRORS
}

// Whether an event has completed.  Also while a graph is being captured, when a plain query would end the capture: the
// event was recorded outside it, and in relaxed mode the question touches nothing that is captured.
PyObject* py_event_done(PyObject*, PyObject* event) {
  HANDLE_TH_ERRORS
  const cudaEvent_t ev = as_event(event);
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  cuda_ok(cudaThreadExchangeStreamCaptureMode(&mode), "cudaThreadExchangeStreamCaptureMode");
  const cudaError_t e = cudaEventQuery(ev);
  const cudaError_t back = cudaThreadExchangeStreamCaptureMode(&mode);
  if (e == cudaErrorNotReady) {
    (void)cudaGetLastError();
    Py_RETURN_FALSE;
  }
  cuda_ok(e, "cudaEventQuery");
  cuda_ok(back, "cudaThreadExchangeStreamCaptureMode");
  Py_RETURN_TRUE;
  END_HANDLE_TH_ERRORS
}

PyObject* py_wait_event(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  want_args(n, 2, "wait_event");
  cuda_ok(cudaStreamWaitEvent(c10::cuda::getCurrentCUDAStream(as_device(a[1])).stream(), as_event(a[0]), 0), "cudaStreamWaitEvent");
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}

// Whether the device's current stream is being captured into a graph
PyObject* py_capturing(PyObject*, PyObject* device) {
  HANDLE_TH_ERRORS
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  const cudaError_t e = cudaStreamIsCapturing(c10::cuda::getCurrentCUDAStream(as_device(device)).stream(), &status);
  if (e == cudaErrorStreamCaptureImplicit) {      // the legacy stream beside a capture on a blocking one: not itself captured
    (void)cudaGetLastError();
    Py_RETURN_FALSE;
  }
  cuda_ok(e, "cudaStreamIsCapturing");
  if (status != cudaStreamCaptureStatusNone) Py_RETURN_TRUE;
  Py_RETURN_FALSE;
  END_HANDLE_TH_ERRORS
}

#define FAST(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_##name)), METH_FASTCALL, nullptr}
PyMethodDef kMethods[] = {FAST(linear_wq), FAST(linear_a4), FAST(conv2d_wq), FAST(conv2d_a4),
                          FAST(hard_quantize), FAST(fake_quantize_ste), FAST(unpack_bits), FAST(pack_bits), FAST(add_layer_norm),
                          FAST(max_pool_nhwc), FAST(images_to_nhwc), FAST(attention_qkv),
                          {"set_launch_count", py_set_launch_count, METH_O, nullptr},
                          {"set_ops", py_set_ops, METH_O, nullptr},
                          {"record_event", py_record_event, METH_O, nullptr},
                          {"event_done", py_event_done, METH_O, nullptr},
                          FAST(wait_event),
                          {"capturing", py_capturing, METH_O, nullptr},
                          {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_host", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host() { return PyModule_Create(&kModule); }
