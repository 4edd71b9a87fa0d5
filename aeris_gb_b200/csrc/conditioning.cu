// Everything around the conditioning vector and the two ends' weights that is too small to be a GEMM: what counts here is
// the number of launches (a training step of a small model was issued in about 275 launches, two thirds of them
// element-wise operations on a few thousand values) and, for wide models, streaming the modulation weights once.
//   * noise_embedding: sinusoidal embedding of the noise level (reference src/aeris/models/parallel_swin.py:61-77)
//   * gemv_bias_act / gemv_bwd: the M <= 8 modulation MLP layers (parallel_swin.py:321-325) and their gradients
//   * pack_embed_weights / fold_embed_grad: [hi(W) | hi(W) | lo(W) | hi(b) | lo(b)] operand of the input projection and
//     the packed product's gradient back on W and b
//   * pack_head_weights: [hi | lo | hi] parts of the output head's weight, padded to a whole number of rows
#include "common.cuh"
#include "api.h"

namespace aeris {

// out[b, :] = [sin(t f_i) | cos(t f_i)], f_i = exp(-ln(max_period) i / half). Double precision: a handful of values, and the
// fast single-precision sine would cost accuracy at large angles.
// `Levels`: where t comes from, an array in memory or one that travels with the launch.
constexpr int MAX_LEVELS = 64;
struct DeviceLevels {
  const float* t;
  __device__ float operator[](int b) const { return t[b]; }
};
struct HostLevels {
  float t[MAX_LEVELS];
  __device__ float operator[](int b) const { return t[b]; }
};
template <typename OT, typename Levels>
__global__ void noise_embedding_kernel(const Levels t, OT* __restrict__ out, int B, int dim, double log_period) {
  const int half = dim / 2;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < B * half; i += gridDim.x * blockDim.x) {
    const int b = i / half, k = i - b * half;
    const double a = static_cast<double>(t[b]) * exp(-log_period * k / half);
    double s, c;
    sincos(a, &s, &c);
    OT* o = out + static_cast<size_t>(b) * dim + k;
    if constexpr (sizeof(OT) == 2) {
      o[0] = __float2bfloat16_rn(static_cast<float>(s));
      o[half] = __float2bfloat16_rn(static_cast<float>(c));
    } else {
      o[0] = static_cast<float>(s);
      o[half] = static_cast<float>(c);
    }
  }
}

template <typename T>
__device__ __forceinline__ float to_f32(T v) {
  if constexpr (sizeof(T) == 2) return __bfloat162float(v); else return v;
}
__device__ __forceinline__ void load_w8(const __nv_bfloat16* p, float (&f)[8]) {
  const uint4 u = *reinterpret_cast<const uint4*>(p);
  const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 t = unpack_bf16x2(w[i]);
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
  }
}
__device__ __forceinline__ void load_w8(const float* p, float (&f)[8]) {
  const float4 a = reinterpret_cast<const float4*>(p)[0], b = reinterpret_cast<const float4*>(p)[1];
  f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w;
  f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
}
__device__ __forceinline__ float load_any(const void* p, size_t i, bool bf16) {
  return bf16 ? __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(p)[i]) : reinterpret_cast<const float*>(p)[i];
}

// Most shared memory that the rows of x (B rounded up to 1, 2, 4 or 8) may take: 8 rows of 6,400 columns, 4 of 12,800.
constexpr int GEMV_X_BYTES = 200 * 1024;

// y[b, n] = act(sum_k W[n, k] silu?(x[b, k]) + bias[n]) for B <= 8 rows: one warp per output feature streams one weight
// row, eight weights (16 bytes of bf16) per lane and load where `vec` says that rows start on 16-byte boundaries. act: 0
// none, 1 SiLU. Bound by the weight stream; MB is B rounded up to 1, 2, 4 or 8. 30720 x 5120 bf16 (B = 1): 281 ->
// 61 us (5.1 TB/s) against two-byte loads.
template <typename WT, int MB>
__global__ void __launch_bounds__(256)
gemv_bias_act_kernel(const WT* __restrict__ W, const void* __restrict__ bias, int bias_bf16, const void* __restrict__ x,
                     int x_bf16, float* __restrict__ y, int N, int K, int B, int act, int silu_in, int vec) {
  chain_point();
  extern __shared__ __align__(16) float xs[];  // [MB, Kp], rows padded to a multiple of four floats
  const int Kp = (K + 3) & ~3;
  for (int b = 0; b < MB; ++b)
    for (int k = threadIdx.x; k < K; k += blockDim.x) {
      float t = 0.f;
      if (b < B) {
        t = load_any(x, static_cast<size_t>(b) * K + k, x_bf16);
        if (silu_in) t = t / (1.f + __expf(-t));
      }
      xs[b * Kp + k] = t;
    }
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (int n = blockIdx.x * nw + warp; n < N; n += gridDim.x * nw) {
    float acc[MB];
#pragma unroll
    for (int b = 0; b < MB; ++b) acc[b] = 0.f;
    const WT* wr = W + static_cast<size_t>(n) * K;
    if (vec) {
#pragma unroll 4
      for (int k = lane * 8; k < K; k += 256) {
        float w[8];
        load_w8(wr + k, w);
#pragma unroll
        for (int b = 0; b < MB; ++b) {
          const float4* xv = reinterpret_cast<const float4*>(xs + b * Kp + k);
          const float4 a = xv[0], c = xv[1];
          acc[b] = fmaf(w[0], a.x, acc[b]); acc[b] = fmaf(w[1], a.y, acc[b]);
          acc[b] = fmaf(w[2], a.z, acc[b]); acc[b] = fmaf(w[3], a.w, acc[b]);
          acc[b] = fmaf(w[4], c.x, acc[b]); acc[b] = fmaf(w[5], c.y, acc[b]);
          acc[b] = fmaf(w[6], c.z, acc[b]); acc[b] = fmaf(w[7], c.w, acc[b]);
        }
      }
    } else {
      for (int k = lane; k < K; k += 32) {
        const float w = to_f32(wr[k]);
#pragma unroll
        for (int b = 0; b < MB; ++b) acc[b] = fmaf(w, xs[b * Kp + k], acc[b]);
      }
    }
#pragma unroll
    for (int b = 0; b < MB; ++b) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) acc[b] += __shfl_xor_sync(0xffffffffu, acc[b], o);
    }
    if (lane == 0) {
      const float bv = bias ? load_any(bias, n, bias_bf16) : 0.f;
#pragma unroll
      for (int b = 0; b < MB; ++b) {
        if (b >= B) break;
        float v = acc[b] + bv;
        if (act == 1) v = v / (1.f + __expf(-v));
        y[static_cast<size_t>(b) * N + n] = v;
      }
    }
  }
}

// Gradients of y = silu?(x) W^T + bias for B <= 8 rows in one pass over W and dW:
//   dW[n, k] += sum_b dy[b, n] h[b, k],  db[n] += sum_b dy[b, n],  dx[b, k] += silu'(x[b, k]) sum_n dy[b, n] W[n, k].
// A thread owns four columns k and walks down the CTA's rows; dx (zeroed by the caller; null: not wanted) is added up
// over the CTAs with vector reductions. Bound by the fp32 gradient, read and written once. Before, this was a rank-B GEMM,
// a product with a bf16 copy of dy, and ten element-wise launches per layer. 30720 x 5120: 426 -> 262 us
// (6.0 TB/s of W and dW); 9216 x 1536, issued from Python: 156 -> 71 us.
constexpr int GEMV_BWD_ROWS = 64;
template <typename WT, int MB>
__global__ void __launch_bounds__(256)
gemv_bwd_kernel(const WT* __restrict__ W, const void* __restrict__ x, int x_bf16, const float* __restrict__ dy,
                float* __restrict__ dW, float* __restrict__ db, float* __restrict__ dx, int N, int K, int B, int silu_in,
                int rows) {
  chain_point();
  __shared__ float s_dy[GEMV_BWD_ROWS][MB];
  const int n0 = blockIdx.y * rows, nr = min(rows, N - n0);
  for (int i = threadIdx.x; i < nr * MB; i += blockDim.x) {
    const int r = i / MB, b = i - r * MB;
    s_dy[r][b] = b < B ? dy[static_cast<size_t>(b) * N + n0 + r] : 0.f;
  }
  __syncthreads();
  if (db && blockIdx.x == 0) {
    for (int r = threadIdx.x; r < nr; r += blockDim.x) {
      float s = 0.f;
#pragma unroll
      for (int b = 0; b < MB; ++b) s += s_dy[r][b];
      db[n0 + r] += s;
    }
  }
  const int k = (blockIdx.x * blockDim.x + threadIdx.x) * 4;
  if (k >= K) return;
  float h[MB][4], dh[MB][4], acc[MB][4];      // silu?(x), silu'(x) or 1, column sums
#pragma unroll
  for (int b = 0; b < MB; ++b)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float v = b < B ? load_any(x, static_cast<size_t>(b) * K + k + i, x_bf16) : 0.f;
      h[b][i] = v;
      dh[b][i] = 1.f;
      acc[b][i] = 0.f;
      if (silu_in) {
        const float s = 1.f / (1.f + __expf(-v));
        h[b][i] = v * s;
        dh[b][i] = s * (1.f + v * (1.f - s));
      }
    }
#pragma unroll 8
  for (int r = 0; r < nr; ++r) {
    const size_t off = static_cast<size_t>(n0 + r) * K + k;
    float4 d = *reinterpret_cast<const float4*>(dW + off);
    float w[4] = {0.f, 0.f, 0.f, 0.f};
    if (dx) {
      if constexpr (sizeof(WT) == 2) {
        const uint2 u = *reinterpret_cast<const uint2*>(W + off);
        const float2 a = unpack_bf16x2(u.x), c = unpack_bf16x2(u.y);
        w[0] = a.x; w[1] = a.y; w[2] = c.x; w[3] = c.y;
      } else {
        const float4 u = *reinterpret_cast<const float4*>(W + off);
        w[0] = u.x; w[1] = u.y; w[2] = u.z; w[3] = u.w;
      }
    }
#pragma unroll
    for (int b = 0; b < MB; ++b) {
      const float g = s_dy[r][b];
      d.x = fmaf(g, h[b][0], d.x); d.y = fmaf(g, h[b][1], d.y);
      d.z = fmaf(g, h[b][2], d.z); d.w = fmaf(g, h[b][3], d.w);
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[b][i] = fmaf(g, w[i], acc[b][i]);
    }
    *reinterpret_cast<float4*>(dW + off) = d;
  }
  if (dx) {
#pragma unroll
    for (int b = 0; b < MB; ++b) {
      if (b >= B) break;
      asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dx + static_cast<size_t>(b) * K + k),
                   "f"(acc[b][0] * dh[b][0]), "f"(acc[b][1] * dh[b][1]), "f"(acc[b][2] * dh[b][2]), "f"(acc[b][3] * dh[b][3])
                   : "memory");
    }
  }
}

// Row d of the input projection's packed operand: [hi(W) | hi(W) | lo(W) | hi(b) | lo(b) | 0...] (bf16, KP columns).
__global__ void pack_embed_weights_kernel(const float* __restrict__ W, const float* __restrict__ b,
                                          __nv_bfloat16* __restrict__ out, int D, int Cin, int KP) {
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < static_cast<long long>(D) * KP;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int d = static_cast<int>(i / KP), j = static_cast<int>(i - static_cast<long long>(d) * KP);
    float v = 0.f;
    if (j < 3 * Cin) {
      const int sec = j / Cin;
      v = W[static_cast<size_t>(d) * Cin + j - sec * Cin];
      if (sec == 2) v -= __bfloat162float(__float2bfloat16_rn(v));
    } else if (j < 3 * Cin + 2) {
      v = b[d];
      if (j > 3 * Cin) v -= __bfloat162float(__float2bfloat16_rn(v));
    }
    out[i] = __float2bfloat16_rn(v);
  }
}
// dW[d, c] += G[d, c] + G[d, Cin + c], db[d] += G[d, 3 Cin].
__global__ void fold_embed_grad_kernel(const float* __restrict__ G, float* __restrict__ dW, float* __restrict__ db, int D,
                                       int Cin, int KP) {
  const long long n = static_cast<long long>(D) * (Cin + 1);
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int d = static_cast<int>(i / (Cin + 1)), c = static_cast<int>(i - static_cast<long long>(d) * (Cin + 1));
    const float* g = G + static_cast<size_t>(d) * KP;
    if (c < Cin) dW[static_cast<size_t>(d) * Cin + c] += g[c] + g[Cin + c];
    else db[d] += g[3 * Cin];
  }
}
// Rows [hi(W) | lo(W) | hi(W)] (bf16, [rows, 3 D]) of the fp32 head weight [C, D]; rows past C are zero.
__global__ void pack_head_weights_kernel(const float* __restrict__ W, __nv_bfloat16* __restrict__ out, int C, int rows,
                                         int D) {
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < static_cast<long long>(rows) * D;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int r = static_cast<int>(i / D), c = static_cast<int>(i - static_cast<long long>(r) * D);
    const float v = r < C ? W[i] : 0.f;
    const __nv_bfloat16 h = __float2bfloat16_rn(v);
    __nv_bfloat16* o = out + static_cast<size_t>(r) * 3 * D + c;
    o[0] = h;
    o[D] = __float2bfloat16_rn(v - __bfloat162float(h));
    o[2 * D] = h;
  }
}

}  // namespace aeris

using namespace aeris;
extern int aeris_num_sms();

static int small_grid(long long n) {
  const long long b = (n + 255) / 256, cap = static_cast<long long>(aeris_num_sms()) * 8;
  return static_cast<int>(b < 1 ? 1 : b > cap ? cap : b);
}
static int launched() { return cudaGetLastError() == cudaSuccess ? 0 : -21; }

template <typename Levels>
static int noise_embedding(const Levels& t, void* out, int out_bf16, int B, int dim, double max_period, void* stream) {
  if (B <= 0 || dim <= 0 || dim % 2 || !(max_period > 0)) return -1;
  const cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const int grid = small_grid(static_cast<long long>(B) * (dim / 2));
  const double lp = log(max_period);
  if (out_bf16) noise_embedding_kernel<<<grid, 256, 0, st>>>(t, reinterpret_cast<__nv_bfloat16*>(out), B, dim, lp);
  else          noise_embedding_kernel<<<grid, 256, 0, st>>>(t, reinterpret_cast<float*>(out), B, dim, lp);
  return launched();
}
extern "C" int aeris_noise_embedding(const float* t, void* out, int out_bf16, int B, int dim, double max_period,
                                     void* stream) {
  return noise_embedding(DeviceLevels{t}, out, out_bf16, B, dim, max_period, stream);
}
extern "C" int aeris_noise_embedding_of(const float* levels, void* out, int out_bf16, int n, int dim, double max_period,
                                        void* stream) {
  if (n <= 0 || n > MAX_LEVELS) return -1;
  HostLevels t = {};
  for (int i = 0; i < n; ++i) t.t[i] = levels[i];
  return noise_embedding(t, out, out_bf16, n, dim, max_period, stream);
}

// flags: 1 = W fp32 (else bf16), 2 = bias bf16 (else fp32), 4 = x bf16 (else fp32)
extern "C" int aeris_gemv_bias_act(const void* W, int flags, const void* bias, const void* x, float* y, int N, int K, int B,
                                   int act, int silu_in, void* stream) {
  if (N <= 0 || K <= 0 || B <= 0 || B > 8) return -1;
  const int mb = B <= 1 ? 1 : B <= 2 ? 2 : B <= 4 ? 4 : 8;
  const size_t smem = static_cast<size_t>(mb) * ((K + 3) & ~3) * sizeof(float);
  if (smem > GEMV_X_BYTES) return -2;
  const int vec = K % 8 == 0 && (reinterpret_cast<uintptr_t>(W) & 15) == 0;
  int grid = (N + 7) / 8;
  const int cap = aeris_num_sms() * 8;
  if (grid > cap) grid = cap;
  const cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
#define AERIS_GEMV(WT, MB)                                                                                              \
  do {                                                                                                                  \
    auto kern = gemv_bias_act_kernel<WT, MB>;                                                                           \
    if (smem > 48 * 1024 &&                                                                                             \
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, GEMV_X_BYTES) != cudaSuccess)           \
      return -20;                                                                                                       \
    return launch_chained(kern, grid, 256, smem, st, reinterpret_cast<const WT*>(W), bias, (flags >> 1) & 1, x,         \
                          (flags >> 2) & 1, y, N, K, B, act, silu_in, vec);                                             \
  } while (0)
#define AERIS_GEMV_MB(WT) \
  do { if (mb == 1) AERIS_GEMV(WT, 1); else if (mb == 2) AERIS_GEMV(WT, 2); \
       else if (mb == 4) AERIS_GEMV(WT, 4); else AERIS_GEMV(WT, 8); } while (0)
  if (flags & 1) AERIS_GEMV_MB(float); else AERIS_GEMV_MB(__nv_bfloat16);
#undef AERIS_GEMV_MB
#undef AERIS_GEMV
}

// The modulation MLP: y1 = x W1^T + b1 [B, N1], y2 = silu(y1) W2^T + b2 [B, N2]. Flags as above, for each layer.
extern "C" int aeris_modulation_mlp(const void* W1, int flags1, const void* b1, const void* x, float* y1, int N1, int K,
                                    const void* W2, int flags2, const void* b2, float* y2, int N2, int B, void* stream) {
  const int rc = aeris_gemv_bias_act(W1, flags1, b1, x, y1, N1, K, B, 0, 0, stream);
  return rc ? rc : aeris_gemv_bias_act(W2, flags2, b2, y1, y2, N2, N1, B, 0, 1, stream);
}

// flags as above. K must be a multiple of 4; W, dW and dx aligned to four elements. dW, db and dx are added to.
extern "C" int aeris_gemv_bwd(const void* W, int flags, const void* x, const float* dy, float* dW, float* db, float* dx,
                              int N, int K, int B, int silu_in, void* stream) {
  if (N <= 0 || K <= 0 || K % 4 || B <= 0 || B > 8 || N > 65535 * 16) return -1;
  if ((reinterpret_cast<uintptr_t>(W) & ((flags & 1) ? 15 : 7)) ||
      ((reinterpret_cast<uintptr_t>(dW) | reinterpret_cast<uintptr_t>(dx)) & 15))
    return -3;
  int nt = (K / 4 + 31) / 32 * 32;
  if (nt > 256) nt = 256;
  // 64 rows per CTA where that still gives every SM four CTAs (fewer reductions into dx), else 16: the walk down the rows is
  // a chain of loads, and a narrow layer spent 35 us in it (1536 x 256; 11 us with 16 rows)
  const int kx = (K / 4 + nt - 1) / nt;
  const int rows = static_cast<long long>(kx) * (N / GEMV_BWD_ROWS) >= 4ll * aeris_num_sms() ? GEMV_BWD_ROWS : 16;
  const dim3 grid(kx, (N + rows - 1) / rows);
  const int mb = B <= 1 ? 1 : B <= 2 ? 2 : B <= 4 ? 4 : 8;
  const cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
#define AERIS_GEMV(WT, MB) \
  return launch_chained(gemv_bwd_kernel<WT, MB>, grid, nt, 0, st, reinterpret_cast<const WT*>(W), x, (flags >> 2) & 1, \
                        dy, dW, db, dx, N, K, B, silu_in, rows)
#define AERIS_GEMV_MB(WT) \
  do { if (mb == 1) AERIS_GEMV(WT, 1); else if (mb == 2) AERIS_GEMV(WT, 2); \
       else if (mb == 4) AERIS_GEMV(WT, 4); else AERIS_GEMV(WT, 8); } while (0)
  if (flags & 1) AERIS_GEMV_MB(float); else AERIS_GEMV_MB(__nv_bfloat16);
#undef AERIS_GEMV_MB
#undef AERIS_GEMV
}

// Gradients of aeris_modulation_mlp, added to dW1, db1, dW2 and db2; dy1 [B, N1] (scratch) and dx [B, K] (may be null) are
// overwritten.
extern "C" int aeris_modulation_mlp_bwd(const void* W1, int flags1, const void* x, float* dW1, float* db1, float* dx, int N1,
                                        int K, const void* W2, int flags2, const float* y1, const float* dy, float* dW2,
                                        float* db2, float* dy1, int N2, int B, void* stream) {
  if (N1 <= 0 || K <= 0 || B <= 0) return -1;
  const cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (cudaMemsetAsync(dy1, 0, sizeof(float) * B * N1, st) != cudaSuccess ||
      (dx && cudaMemsetAsync(dx, 0, sizeof(float) * B * K, st) != cudaSuccess))
    return -20;
  const int rc = aeris_gemv_bwd(W2, flags2, y1, dy, dW2, db2, dy1, N2, N1, B, 1, stream);
  return rc ? rc : aeris_gemv_bwd(W1, flags1, x, dy1, dW1, db1, dx, N1, K, B, 0, stream);
}

extern "C" int aeris_pack_embed_weights(const float* W, const float* b, void* out, int D, int Cin, int KP, void* stream) {
  if (D <= 0 || Cin <= 0 || KP < 3 * Cin + 2) return -1;
  pack_embed_weights_kernel<<<small_grid(static_cast<long long>(D) * KP), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      W, b, reinterpret_cast<__nv_bfloat16*>(out), D, Cin, KP);
  return launched();
}

extern "C" int aeris_fold_embed_grad(const float* G, float* dW, float* db, int D, int Cin, int KP, void* stream) {
  if (D <= 0 || Cin <= 0 || KP < 3 * Cin + 2) return -1;
  const int grid = small_grid(static_cast<long long>(D) * (Cin + 1));
  fold_embed_grad_kernel<<<grid, 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(G, dW, db, D, Cin, KP);
  return launched();
}

extern "C" int aeris_pack_head_weights(const float* W, void* out, int C, int rows, int D, void* stream) {
  if (C <= 0 || rows < C || D <= 0) return -1;
  pack_head_weights_kernel<<<small_grid(static_cast<long long>(rows) * D), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      W, reinterpret_cast<__nv_bfloat16*>(out), C, rows, D);
  return launched();
}
