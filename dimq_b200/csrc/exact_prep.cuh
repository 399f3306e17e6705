// Operand preparation of the fp32-grade GEMM / convolution (the SEG form of lut_dense_tc_kernel): ONE kernel
// turns the activations into fp16 operands and expands the packed weight, so the product that follows costs two
// launches in all.
//
// Why fp16 terms.  The tensor cores multiply 16-bit operands exactly and add in fp32.
//   * W4A4: the activation codes minus their zero point are integers in [-15, 15], exact in fp16.
//   * fp32 activations: x * 2^e = hi + lo * 2^-12 with fp16 hi and lo; e is chosen per row so that the row's largest
//     finite magnitude lies in [2^14, 2^15).  hi carries 11 bits, lo the next 11 and the sign of lo one more: about 2^-23
//     of the element.  lo is stored 2^12 times as large, so that it has its bits left where hi comes to fp16's end: an
//     element keeps 2^-23 down to 2^-28 of the row's largest and is known to 2^-51 of that below.  (With lo as it is,
//     the range ended at 2^-18: rows of order 1 with one element of 1e8 that meets a zero codeword came out at 6.8e-5.)
//     The sums of the products with a lo are taken out of the accumulators apart and multiplied by 2^-12.
//   * codewords: fp16 ones are their own term.  Others are scaled per group in the same way; bf16 ones (8 bits, exact down
//     to 2^-30 of the group's largest) are then one term, fp32 ones hi + lo.
// Three products (x_hi w_hi, x_hi w_lo, x_lo w_hi) carry an fp32 product to about 2^-23; a bf16 split would need six.
// Non-finite values of the fp32 form: an infinite activation has hi = 0 and keeps its value in lo, which meets w_hi only; a
// codeword that would underflow to w_hi = 0 takes fp16's smallest instead (w_lo carries the difference), so the product has
// the sign of both.  A row with a NaN has the scale NaN.  An infinite or NaN codeword is a NaN here: no split of it is right,
// as x_lo may be zero, or of the other sign, where x is not.  Where an output of such a codebook comes out as a NaN and its
// row has none, the epilogue computes it again in plain fp32.
// W4A4 codes are one exact term: a zero code against an infinite codeword is NaN as in fp32, with one term or two (there
// w_lo keeps the value and w_hi = 0).
#pragma once

#include "common.cuh"

namespace dimq {
namespace {

constexpr int kPrepThreads = 256;
constexpr float kLoScale = 4096.0f;      // lo terms are stored this many times as large (the SEG epilogue divides)
constexpr int kExpandTable = 129 * 16;   // words: a block of 256 units covers at most 128 rows (K >= 64), 129 groups

// exponent e with max_abs * 2^e in [2^14, 2^15), kept where 2^-e is a normal number: max_abs below 2^-112 is scaled by 2^126,
// which takes the smallest subnormal to 2^-23, still a multiple of fp16's smallest.  The product of a row's and a column's
// 2^-e may leave fp32; the epilogue multiplies by one after the other.
__device__ __forceinline__ int fp16_scale_exponent(float max_abs) {
  if (!(max_abs > 0.0f)) return 0;
  const int e = 14 - ilogbf(max_abs);
  return e > 126 ? 126 : e;
}

__device__ __forceinline__ bool finite_f32(float v) { return fabsf(v) <= 3.402823466e38f; }

// lut_expand_kernel's work for one block of 256 units (unit = 32 consecutive indices of one row).
//   fmt 0: fp16 codewords, 1: bf16 (terms == 2: and the bf16 remainder c - bf16(c)), 2: fp16 of c * 2^e with e per
//   group (terms == 2: and the fp16 remainder times kLoScale); col_scale[row] = 2^-e.
//   split_x: for activations in two terms, see above (fmt 0 and 2).
template <int BITS>
__device__ __forceinline__ void expand_block(uint32_t* tbl, int64_t block, const uint8_t* __restrict__ packed,
                                             const void* __restrict__ codebooks, int cb_dtype, int entries,
                                             int64_t group_rows, int64_t rows, int64_t K, int fmt, int terms,
                                             uint16_t* __restrict__ out, float* __restrict__ col_scale, bool split_x) {
  const int64_t units_per_row = K / 32;
  const int64_t total = rows * units_per_row;
  const int64_t u = block * 256 + threadIdx.x;
  // Up to 16-entry codebooks: the codewords of the groups this block's rows belong to are converted once
  // into a shared-memory table (hi | lo << 16), so an index costs one shared-memory read instead of a global
  // read and two conversions.
  constexpr bool kTable = BITS <= 4;
  int64_t g_first = 0;
  if (kTable) {
    const int64_t u_first = block * 256;
    const int64_t u_last = u_first + 255 < total - 1 ? u_first + 255 : total - 1;
    g_first = (u_first / units_per_row) / group_rows;
    const int n_slots = (static_cast<int>((u_last / units_per_row) / group_rows - g_first) + 1) * 16;
    for (int i0 = 0; i0 < n_slots; i0 += 256) {       // whole warps stay in the loop: the 16 lanes of a group share its scale
      const int i = i0 + threadIdx.x;
      const int e = i & 15;
      const int64_t g = g_first + (i >> 4);
      const float c = i < n_slots && e < entries ? load_as_float(codebooks, cb_dtype, g * entries + e) : 0.0f;
      uint32_t v;
      if (fmt == 0) {
        v = split_x && !finite_f32(c) ? 0x7FFFu : __half_as_ushort(__float2half_rn(c));
      } else if (fmt == 1) {
        const __nv_bfloat16 h = __float2bfloat16_rn(c);
        v = __bfloat16_as_ushort(h) | (static_cast<uint32_t>(__bfloat16_as_ushort(__float2bfloat16_rn(c - __bfloat162float(h)))) << 16);
      } else {
        float mx = finite_f32(c) ? fabsf(c) : 0.0f;
#pragma unroll
        for (int d = 8; d > 0; d >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, d));
        const int ex = fp16_scale_exponent(mx);
        const float cs = scalbnf(c, ex);
        __half h = __float2half_rn(cs), l = __float2half_rn(0.0f);
        if (split_x && !finite_f32(c)) {
          h = __ushort_as_half(0x7FFFu);
        } else if (split_x && c != 0.0f && fabsf(cs) <= 2.98023224e-8f) {   // 2^-25
          h = __float2half_rn(copysignf(5.96046448e-8f, c));
        }
        if (terms == 2) {
          if (finite_f32(c)) l = __float2half_rn((cs - __half2float(h)) * kLoScale);
          else if (!split_x) { l = h; h = __float2half_rn(0.0f); }
        }
        v = __half_as_ushort(h) | (static_cast<uint32_t>(__half_as_ushort(l)) << 16);
        // the scale of every row of this group that starts in this block's units (first unit of the row)
        if (e == 0 && i < n_slots) {
          const float inv = scalbnf(1.0f, -ex);
          const int64_t r_lo = (u_first + units_per_row - 1) / units_per_row, r_hi = u_last / units_per_row;
          int64_t r = g * group_rows > r_lo ? g * group_rows : r_lo;
          const int64_t r_end = (g + 1) * group_rows - 1 < r_hi ? (g + 1) * group_rows - 1 : r_hi;
          for (; r <= r_end; ++r) col_scale[r] = inv;
        }
      }
      if (i < n_slots) tbl[i] = v;
    }
    __syncthreads();
  }
  if (u >= total) return;
  const int64_t row = u / units_per_row;
  const int64_t k0 = (u - row * units_per_row) * 32;
  const uint32_t* src = reinterpret_cast<const uint32_t*>(packed + (row * K + k0) * BITS / 8);
  uint32_t w[BITS];
#pragma unroll
  for (int i = 0; i < BITS; ++i) w[i] = __ldg(src + i);
  const int64_t cb0 = (row / group_rows) * entries;
  const uint32_t* my_tbl = tbl + (kTable ? static_cast<int>(row / group_rows - g_first) * 16 : 0);
  uint16_t hi[32], lo[32];
#pragma unroll
  for (int i = 0; i < 32; ++i) {
    const int bit = i * BITS, word = bit >> 5, sh = bit & 31;
    uint32_t idx = w[word] >> sh;
    if (sh + BITS > 32) idx |= w[word + 1 < BITS ? word + 1 : word] << (32 - sh);
    idx &= (1u << BITS) - 1u;
    if (kTable) {
      const uint32_t v = my_tbl[idx];      // entries past the codebook's count hold zero
      hi[i] = static_cast<uint16_t>(v);
      lo[i] = static_cast<uint16_t>(v >> 16);
    } else {
      const float c = idx < static_cast<uint32_t>(entries) ? load_as_float(codebooks, cb_dtype, cb0 + idx) : 0.0f;
      if (fmt == 0) {
        hi[i] = __half_as_ushort(__float2half_rn(c));
        lo[i] = 0;
      } else {
        const __nv_bfloat16 h = __float2bfloat16_rn(c);
        hi[i] = __bfloat16_as_ushort(h);
        lo[i] = __bfloat16_as_ushort(__float2bfloat16_rn(c - __bfloat162float(h)));
      }
    }
  }
  uint16_t* dst = out + row * (K * terms) + k0;
#pragma unroll
  for (int v = 0; v < 4; ++v) {
    uint4 q;
    q.x = hi[8 * v] | (static_cast<uint32_t>(hi[8 * v + 1]) << 16);
    q.y = hi[8 * v + 2] | (static_cast<uint32_t>(hi[8 * v + 3]) << 16);
    q.z = hi[8 * v + 4] | (static_cast<uint32_t>(hi[8 * v + 5]) << 16);
    q.w = hi[8 * v + 6] | (static_cast<uint32_t>(hi[8 * v + 7]) << 16);
    reinterpret_cast<uint4*>(dst)[v] = q;
  }
  if (terms == 2) {
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      uint4 q;
      q.x = lo[8 * v] | (static_cast<uint32_t>(lo[8 * v + 1]) << 16);
      q.y = lo[8 * v + 2] | (static_cast<uint32_t>(lo[8 * v + 3]) << 16);
      q.z = lo[8 * v + 4] | (static_cast<uint32_t>(lo[8 * v + 5]) << 16);
      q.w = lo[8 * v + 6] | (static_cast<uint32_t>(lo[8 * v + 7]) << 16);
      reinterpret_cast<uint4*>(dst + K)[v] = q;
    }
  }
}

// Activation side of the preparation.
enum PrepMode { kPrepSplitRows = 0, kPrepCodes = 1, kPrepCodesNchw = 2, kPrepScaleRows = 3 };

struct PrepParams {
  // activations
  int mode;
  const void* x;
  int x_dtype;
  int vec_ok;                // x is 16-byte aligned
  int64_t n;                 // kPrepCodes: elements; kPrepSplitRows, kPrepScaleRows: rows
  int64_t C, HW;             // kPrepSplitRows, kPrepScaleRows: C = row length; kPrepCodesNchw: channels, pixels per image
  float scale;
  int zp;
  __half* xo;                // codes, or [rows][hi C | lo C]
  float* row_scale;          // kPrepSplitRows, kPrepScaleRows: 2^-e per row
  int64_t x_blocks;          // blocks [0, x_blocks) prepare activations, the rest the weight
  int64_t px_tiles;          // kPrepCodesNchw: ceil(HW / 32)
  // weight
  const uint8_t* packed;
  const void* codebooks;
  int cb_dtype, entries;
  int64_t group_rows, rows, K;
  int fmt, terms, split_x;   // see expand_block
  uint16_t* wo;
  float* col_scale;
};

__device__ __forceinline__ __half code_half(float x, float scale, int zp) {
  return __float2half_rn(static_cast<float>(static_cast<int>(quantize_u4(x, scale, zp)) - zp));
}

// 8 consecutive elements as floats (16-byte loads)
__device__ __forceinline__ void load8(const void* x, int dtype, int64_t i, float (&f)[8]) {
  if (dtype == DIMQ_F32) {
    const float4 a = __ldg(reinterpret_cast<const float4*>(static_cast<const float*>(x) + i));
    const float4 b = __ldg(reinterpret_cast<const float4*>(static_cast<const float*>(x) + i) + 1);
    f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
  } else {
    const uint4 q = __ldg(reinterpret_cast<const uint4*>(static_cast<const uint16_t*>(x) + i));
    const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 v = dtype == DIMQ_F16 ? __half22float2(*reinterpret_cast<const __half2*>(&w[j]))
                                         : __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w[j]));
      f[2 * j] = v.x; f[2 * j + 1] = v.y;
    }
  }
}

// One block: activations of its share, or 256 units of the weight.  The two are independent, so a small call pays
// one launch for both and the wide activation pass of a large one hides the lookups.
template <int BITS>
__global__ void __launch_bounds__(kPrepThreads)
exact_prep_kernel(const PrepParams p) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");   // the GEMM's prologue may start; it waits before it reads
  __shared__ __align__(16) uint32_t smem[kExpandTable];
  const int tid = threadIdx.x;
  const int64_t blk = blockIdx.x;
  if (blk >= p.x_blocks) {
    expand_block<BITS>(smem, blk - p.x_blocks, p.packed, p.codebooks, p.cb_dtype, p.entries, p.group_rows, p.rows, p.K,
                       p.fmt, p.terms, p.wo, p.col_scale, p.split_x != 0);
    return;
  }
  if (p.mode == kPrepCodes) {
    const int64_t base = (blk * kPrepThreads + tid) * 8;
    if (base >= p.n) return;
    if (p.vec_ok && base + 8 <= p.n) {
      float f[8];
      load8(p.x, p.x_dtype, base, f);
      __align__(16) __half o[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) o[i] = code_half(f[i], p.scale, p.zp);
      *reinterpret_cast<uint4*>(p.xo + base) = *reinterpret_cast<const uint4*>(o);
    } else {
      for (int i = 0; i < 8 && base + i < p.n; ++i) p.xo[base + i] = code_half(load_as_float(p.x, p.x_dtype, base + i), p.scale, p.zp);
    }
  } else if (p.mode == kPrepCodesNchw) {
    // 64 channels x 32 pixels through shared memory: a warp reads 32 consecutive pixels of one channel, a thread
    // writes 8 channels of one pixel (16 bytes).  Row pitch 33 words: neither side has a bank conflict.
    __half* tile = reinterpret_cast<__half*>(smem);
    const int64_t px0 = (blk % p.px_tiles) * 32;
    const int64_t c0 = ((blk / p.px_tiles) % (p.C / 64)) * 64;
    const int64_t b = blk / (p.px_tiles * (p.C / 64));
    const int lane = tid & 31, warp = tid >> 5;
    const int64_t px = px0 + lane;
    const bool in = px < p.HW;
    float f[8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
      f[i] = in ? load_as_float(p.x, p.x_dtype, (b * p.C + c0 + warp * 8 + i) * p.HW + px) : 0.0f;
#pragma unroll
    for (int i = 0; i < 8; ++i) tile[lane * 66 + warp * 8 + i] = code_half(f[i], p.scale, p.zp);
    __syncthreads();
    const int my_px = tid >> 3, cg = tid & 7;
    if (px0 + my_px < p.HW) {
      const uint32_t* src = smem + my_px * 33 + cg * 4;
      *reinterpret_cast<uint4*>(p.xo + (b * p.HW + px0 + my_px) * p.C + c0 + cg * 8) = make_uint4(src[0], src[1], src[2], src[3]);
    }
  } else if (p.mode == kPrepScaleRows) {
    // bf16 rows -> fp16(x * 2^e), two rows per block, four warps each (infinities and NaN stay what they are)
    const int half_id = tid >> 7, t = tid & 127;
    const int64_t row = blk * 2 + half_id;
    const bool live = row < p.n;
    const uint16_t* xr = static_cast<const uint16_t*>(p.x) + (live ? row : 0) * p.C;
    float mx = 0.0f;
    if (live)
      for (int64_t k = t * 8; k < p.C; k += 1024) {     // C % 64 == 0
        float f[8];
        load8(xr, DIMQ_BF16, k, f);
#pragma unroll
        for (int i = 0; i < 8; ++i) mx = fmaxf(mx, finite_f32(f[i]) ? fabsf(f[i]) : 0.0f);
      }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, d));
    if ((tid & 31) == 0) smem[tid >> 5] = __float_as_uint(mx);
    __syncthreads();
    if (!live) return;
#pragma unroll
    for (int i = 0; i < 4; ++i) mx = fmaxf(mx, __uint_as_float(smem[half_id * 4 + i]));
    const int ex = fp16_scale_exponent(mx);
    if (t == 0) p.row_scale[row] = scalbnf(1.0f, -ex);
    const float up = scalbnf(1.0f, ex);      // -113 <= ex <= 126: a normal number
    for (int64_t k = t * 8; k < p.C; k += 1024) {
      float f[8];
      load8(xr, DIMQ_BF16, k, f);
      __align__(16) __half o[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) o[i] = __float2half_rn(f[i] * up);
      *reinterpret_cast<uint4*>(p.xo + row * p.C + k) = *reinterpret_cast<const uint4*>(o);
    }
  } else {
    // two rows per block, four warps each: the row's largest finite magnitude, then hi and lo (the second read of
    // the row comes from L1)
    const int half_id = tid >> 7, t = tid & 127;
    const int64_t row = blk * 2 + half_id;
    const bool live = row < p.n;
    const float* xr = static_cast<const float*>(p.x) + (live ? row : 0) * p.C;
    float mx = 0.0f;
    bool nan = false;
    if (live)
      for (int64_t k = t * 4; k < p.C; k += 512) {      // C % 64 == 0
        const float4 v = __ldg(reinterpret_cast<const float4*>(xr + k));
        const float a[4] = {fabsf(v.x), fabsf(v.y), fabsf(v.z), fabsf(v.w)};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          mx = fmaxf(mx, finite_f32(a[i]) ? a[i] : 0.0f);
          nan = nan || a[i] != a[i];
        }
      }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, d));
    nan = __any_sync(0xFFFFFFFFu, nan);
    if ((tid & 31) == 0) { smem[tid >> 5] = __float_as_uint(mx); smem[8 + (tid >> 5)] = nan ? 1u : 0u; }
    __syncthreads();
    if (!live) return;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      mx = fmaxf(mx, __uint_as_float(smem[half_id * 4 + i]));
      nan = nan || smem[8 + half_id * 4 + i] != 0u;
    }
    const int ex = fp16_scale_exponent(mx);
    if (t == 0) p.row_scale[row] = nan ? __int_as_float(0x7FFFFFFF) : scalbnf(1.0f, -ex);
    const float up = scalbnf(1.0f, ex);      // -113 <= ex <= 126: a normal number
    __half* hi = p.xo + row * 2 * p.C;
    for (int64_t k = t * 4; k < p.C; k += 512) {
      const float4 v = __ldg(reinterpret_cast<const float4*>(xr + k));
      const float a[4] = {v.x, v.y, v.z, v.w};
      __align__(8) __half h[4], l[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float s = a[i] * up;
        if (finite_f32(a[i])) {
          h[i] = __float2half_rn(s);
          l[i] = __float2half_rn((s - __half2float(h[i])) * kLoScale);
        } else {
          h[i] = __float2half_rn(0.0f);
          l[i] = __float2half_rn(a[i]);
        }
      }
      *reinterpret_cast<uint2*>(hi + k) = *reinterpret_cast<const uint2*>(h);
      *reinterpret_cast<uint2*>(hi + p.C + k) = *reinterpret_cast<const uint2*>(l);
    }
  }
}

}  // namespace
}  // namespace dimq
