// Softmax attention over a packed qkv projection, for the whole-model harness: qkv is [B][T][3][H][64] as the qkv Linear
// writes it, the output [B][T][H][64] as the projection reads it - no split, permute or transpose around it.
//
// One block per 64 query rows of one head: K and V of the head (T <= 512 rows of 128 bytes) are copied to shared memory
// once, each of the four warps keeps 16 query rows and walks the keys in chunks of 64 with the running maximum and sum
// of the row (fp32), scores and outputs in warp-level MMA accumulators (fp32), probabilities rounded to the element type
// for the second product, as the library kernels do.  Rows are stored with their 16-byte pieces permuted by row & 7, so
// that neither the copies nor ldmatrix (plain for K, transposed for V) meet a bank conflict.
// What bounds it: one image of 197 tokens and 12 heads has 48 blocks, each a chain of copies, MMAs and reductions (5.3 us;
// scaled_dot_product_attention 6.5, and the view / permute / transpose calls around it cost the host ~20 us more).  A large
// batch is bound by the warp-level MMA rate: 107 us at 128 images where the library's tcgen05 kernel takes 52, so
// the harness uses this one for small batches only.
#include "common.cuh"

namespace dimq {
namespace {

constexpr int kThreads = 128;
constexpr int kD = 64;                 // head dimension: one 128-byte row
constexpr int kQ = 64;                 // query rows per block
constexpr int kChunk = 64;             // keys per step
constexpr int kMaxT = 512;

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool ok) {   // zero-filled where !ok
  const int n = ok ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], uint32_t a) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}
__device__ __forceinline__ void ldsm4_t(uint32_t (&r)[4], uint32_t a) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}

template <bool BF16>
__device__ __forceinline__ void mma16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  if (BF16)
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  else
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

template <bool BF16>
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
  uint32_t d;
  if (BF16) asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo));
  else asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo));
  return d;
}

// byte offset of 16-byte piece c (0..7) of row r in a tile of 128-byte rows
__device__ __forceinline__ uint32_t piece(int r, int c) { return static_cast<uint32_t>(r * 128 + ((c ^ (r & 7)) << 4)); }

template <bool BF16>
__global__ void __launch_bounds__(kThreads)
attention_qkv_kernel(const uint16_t* __restrict__ qkv, uint16_t* __restrict__ out, int T, int H, float scale_log2e) {
  extern __shared__ __align__(128) unsigned char smem[];     // Q 64 rows | K tp rows | V tp rows, tp = T rounded up to 64
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int h = blockIdx.y, q0 = blockIdx.x * kQ;
  const int tp = (T + kChunk - 1) / kChunk * kChunk;
  const int64_t pitch = static_cast<int64_t>(3) * H * kD;
  const uint16_t* base = qkv + static_cast<int64_t>(blockIdx.z) * T * pitch + h * kD;
  const uint32_t sq = smem_addr(smem), sk = sq + kQ * 128, sv = sk + static_cast<uint32_t>(tp) * 128;
  for (int i = tid; i < kQ * 8; i += kThreads) {
    const int r = i >> 3, c = i & 7;
    const bool ok = q0 + r < T;
    cp_async16(sq + piece(r, c), base + static_cast<int64_t>(ok ? q0 + r : 0) * pitch + c * 8, ok);
  }
  for (int i = tid; i < tp * 8; i += kThreads) {
    const int r = i >> 3, c = i & 7;
    cp_async16(sk + piece(r, c), base + static_cast<int64_t>(r < T ? r : 0) * pitch + H * kD + c * 8, r < T);
  }
  cp_async_commit();
  for (int i = tid; i < tp * 8; i += kThreads) {
    const int r = i >> 3, c = i & 7;
    cp_async16(sv + piece(r, c), base + static_cast<int64_t>(r < T ? r : 0) * pitch + 2 * H * kD + c * 8, r < T);
  }
  cp_async_commit();
  cp_async_wait<1>();
  __syncthreads();

  // ldmatrix addresses: lanes 0-7 / 8-15 / 16-23 / 24-31 give the rows of the four 8 x 8 matrices
  const int lr = lane & 7, lm = lane >> 3;
  uint32_t qf[4][4];
#pragma unroll
  for (int ks = 0; ks < 4; ++ks) ldsm4(qf[ks], sq + piece(warp * 16 + lr + (lm & 1) * 8, 2 * ks + (lm >> 1)));

  float o[8][4], mx[2] = {-INFINITY, -INFINITY}, sum[2] = {0.0f, 0.0f};
#pragma unroll
  for (int n = 0; n < 8; ++n) o[n][0] = o[n][1] = o[n][2] = o[n][3] = 0.0f;
  for (int k0 = 0; k0 < T; k0 += kChunk) {
    float s[8][4];
#pragma unroll
    for (int n = 0; n < 8; ++n) s[n][0] = s[n][1] = s[n][2] = s[n][3] = 0.0f;
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) {
#pragma unroll
      for (int np = 0; np < 4; ++np) {      // 16 keys: matrices (keys 0-7, d 0-7), (0-7, 8-15), (8-15, 0-7), (8-15, 8-15)
        uint32_t b[4];
        ldsm4(b, sk + piece(k0 + np * 16 + lr + (lm >> 1) * 8, 2 * ks + (lm & 1)));
        mma16816<BF16>(s[2 * np], qf[ks], b[0], b[1]);
        mma16816<BF16>(s[2 * np + 1], qf[ks], b[2], b[3]);
      }
    }
    if (k0 + kChunk > T) {
#pragma unroll
      for (int n = 0; n < 8; ++n) {
        const int key = k0 + n * 8 + (lane & 3) * 2;
        if (key >= T) s[n][0] = s[n][2] = -INFINITY;
        if (key + 1 >= T) s[n][1] = s[n][3] = -INFINITY;
      }
    }
    // rows lane / 4 and lane / 4 + 8 of the warp's tile; four lanes share a row
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      float m = mx[half];
#pragma unroll
      for (int n = 0; n < 8; ++n) m = fmaxf(m, fmaxf(s[n][2 * half], s[n][2 * half + 1]));
      m = fmaxf(m, __shfl_xor_sync(0xFFFFFFFFu, m, 1));
      m = fmaxf(m, __shfl_xor_sync(0xFFFFFFFFu, m, 2));
      const float ms = m == -INFINITY ? 0.0f : m * scale_log2e;
      const float fix = exp2f(mx[half] * scale_log2e - ms);
      mx[half] = m;
      float part = 0.0f;
#pragma unroll
      for (int n = 0; n < 8; ++n) {
        s[n][2 * half] = exp2f(fmaf(s[n][2 * half], scale_log2e, -ms));
        s[n][2 * half + 1] = exp2f(fmaf(s[n][2 * half + 1], scale_log2e, -ms));
        part += s[n][2 * half] + s[n][2 * half + 1];
        o[n][2 * half] *= fix;
        o[n][2 * half + 1] *= fix;
      }
      sum[half] = sum[half] * fix + part;
    }
    if (k0 == 0) {
      cp_async_wait<0>();
      __syncthreads();
    }
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) {        // 16 keys
      const uint32_t a[4] = {pack2<BF16>(s[2 * ks][0], s[2 * ks][1]), pack2<BF16>(s[2 * ks][2], s[2 * ks][3]),
                             pack2<BF16>(s[2 * ks + 1][0], s[2 * ks + 1][1]), pack2<BF16>(s[2 * ks + 1][2], s[2 * ks + 1][3])};
#pragma unroll
      for (int np = 0; np < 4; ++np) {      // 16 output columns: matrices (keys 0-7, d 0-7), (8-15, 0-7), (0-7, 8-15), (8-15, 8-15)
        uint32_t b[4];
        ldsm4_t(b, sv + piece(k0 + ks * 16 + lr + (lm & 1) * 8, 2 * np + (lm >> 1)));
        mma16816<BF16>(o[2 * np], a, b[0], b[1]);
        mma16816<BF16>(o[2 * np + 1], a, b[2], b[3]);
      }
    }
  }
  // normalise; through this warp's 16 rows of the Q tile (it alone reads them) so that the stores are 16 bytes wide
  __syncwarp();
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    float l = sum[half];
    l += __shfl_xor_sync(0xFFFFFFFFu, l, 1);
    l += __shfl_xor_sync(0xFFFFFFFFu, l, 2);
    const float inv = 1.0f / l;
    const int r = warp * 16 + (lane >> 2) + half * 8;
#pragma unroll
    for (int n = 0; n < 8; ++n)
      *reinterpret_cast<uint32_t*>(smem + piece(r, n) + (lane & 3) * 4) = pack2<BF16>(o[n][2 * half] * inv, o[n][2 * half + 1] * inv);
  }
  __syncwarp();
  uint16_t* dst = out + (static_cast<int64_t>(blockIdx.z) * T * H + h) * kD;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = warp * 16 + i * 4 + (lane >> 3), c = lane & 7;
    if (q0 + r < T)
      *reinterpret_cast<uint4*>(dst + static_cast<int64_t>(q0 + r) * H * kD + c * 8) = *reinterpret_cast<const uint4*>(smem + piece(r, c));
  }
}

}  // namespace
}  // namespace dimq

using namespace dimq;

extern "C" int dimq_attention_qkv(const void* qkv, void* out, int64_t batch, int64_t tokens, int64_t heads, int64_t head_dim,
                                  float scale, int dtype, void* stream) {
  if (batch < 0 || tokens < 0 || heads <= 0) return DIMQ_ERR_BAD_SIZE;
  if (dtype != DIMQ_BF16 && dtype != DIMQ_F16) return DIMQ_ERR_BAD_DTYPE;
  if (head_dim != kD || tokens > kMaxT) return DIMQ_ERR_UNSUPPORTED;
  if (batch > 65535 || heads > 65535) return DIMQ_ERR_TOO_LARGE;
  if (batch == 0 || tokens == 0) return DIMQ_OK;
  if (qkv == nullptr || out == nullptr) return DIMQ_ERR_NULL_POINTER;
  if (!aligned(qkv, 16) || !aligned(out, 16)) return DIMQ_ERR_ALIGNMENT;
  const int tp = static_cast<int>((tokens + kChunk - 1) / kChunk * kChunk);
  const size_t smem = static_cast<size_t>(kQ + 2 * tp) * 128;
  auto kern = dtype == DIMQ_BF16 ? attention_qkv_kernel<true> : attention_qkv_kernel<false>;
  // the kernel's largest, not this call's: the attribute belongs to the process, and another thread's smaller call between
  // this line and the launch would take the limit away again
  const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (kQ + 2 * kMaxT) * 128);
  if (e != cudaSuccess) return static_cast<int>(e);
  const dim3 grid(static_cast<unsigned>((tokens + kQ - 1) / kQ), static_cast<unsigned>(heads), static_cast<unsigned>(batch));
  kern<<<grid, kThreads, smem, static_cast<cudaStream_t>(stream)>>>(static_cast<const uint16_t*>(qkv), static_cast<uint16_t*>(out),
                                                                     static_cast<int>(tokens), static_cast<int>(heads),
                                                                     scale * 1.4426950408889634f);
  return launch_status();
}
